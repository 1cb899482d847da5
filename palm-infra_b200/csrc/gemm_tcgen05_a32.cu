// W4G128 x int8 GEMM on tcgen05.mma kind::i8 under the reference's rule for several rows: one
// activation scale per 32 values (kernels/matmul_w4.cpp:785-901 with the per-32 quantiser,
// kernels/matmul_quant.cpp:280-329).  Per 32-k block b of a group
//   D_b = sum q4*q8 over the block;  y = fma(float(D_b), fp32(ws*as[g][b]), y)
// blocks ascending inside groups ascending.  A block is exactly one K = 32 MMA step, so every
// step has an accumulator of its own and the fp32 chain takes four steps per group.
//
// What bounds it: the issue slots and the fp32 pipe of that chain (M*N*K/32 sums); the MMAs
// keep the tensor pipe under a tenth busy.  So everything around the chain is kept out of it:
//   epilogue   sixteen warps, thread = one token x a quarter of the tile's columns, four warps per
//              scheduler so that one folds while another fetches; a tile of up to 128 columns
//              (row_tiles) spreads what a group costs beside its columns.
//   operands   four warps, every fourth group each, whole groups, its MMAs included.  A nibble
//              becomes a signed byte of 16 q with one AND (high nibble) or a shift and an AND (low
//              nibble): three instructions per eight weights, so the sums are 16 D, |16 D| < 2^19.
//   to float   the hardware conversion, so that the fp32 pipe sees only the scale product and
//              the multiply-add, both paired (fma.rn.f32x2).  It also moves the sums from the
//              registers that the fetch filled to register pairs.  The scales are staged as
//              w / 16: a power of two, exact while w * as / 16 is a normal number.
//   sums       units of half a group, two or four of them in tensor memory; one barrier frees an
//              activation and a weight stage together.
// Measured, 1000 rows, [4100, 9728], three matmuls: tiles of at most 64 columns 882 us; of up to
// 128 with eight epilogue warps and all unpack warps on one group 715 us; this form 613 us.  At 112
// columns a group takes 2180 cycles (clock64, 1.80 GHz): the chain alone, no waits and no other
// warps, 1830 (conversions 448 of a scheduler's issue slots and 896 cycles of its pipe, paired
// products and multiply-adds 224 each and 1140 cycles of the fp32 pipe, fetches 360 on top of
// them); the operand warps beside it 180, the MMAs nothing, waits 170.
// MMAs issued by the warp that unpacks the group, against one warp for the MMAs and three that
// unpack: 40 rows of [2560, 9728] 41.7 -> 36.4 us, 256 rows 53.3 -> 49.7, of [2560, 4096] 25.7 ->
// 24.1, of [19456, 2560] 73.9 -> 73.3, 64 rows of [9728, 2560] 23.6 -> 21.6.
// Tried on the form before: waits that poll in a loop of four instructions, or with test_wait,
// 206 -> 221 us a matmul and 42 -> 62 at 40 rows (pollers take issue slots); hand-over through named
// barriers 235; units of one block 217; the next chunk's fetch under a chunk's sums: no gain.
// Tokens sit on the MMA's M side (128 per CTA), weight rows on its N side.  The next launch
// is released at the start (programmatic dependent launch): weights and scales are fetched
// while the quantiser in front still runs.  Every wait is bounded; on a timeout the kernel
// flags the status word and drains.
#include <utility>

#include "tcgen05_ops.cuh"

namespace {

// Roles: four warps that bring a group's operands in and issue its MMAs, a group in turn, then
// sixteen epilogue warps (four column quarters x four TMEM lane quarters; a warp's lane quarter is
// its index mod 4).  640 threads start with 96 registers each; the epilogue's four warpgroups take
// what the first one gives up.
constexpr int kFeedWarps = 4;
constexpr int kEpiWarp0 = kFeedWarps, kEpiWarps = 16;
constexpr int kThreads = (kEpiWarp0 + kEpiWarps) * 32;
constexpr int kRegsStart = 96, kRegsEpi = 104, kRegsOther = 64;
static_assert(kRegsOther + 4 * kRegsEpi <= 5 * kRegsStart, "registers of the block");
constexpr int kMaxG = 80;  // K <= 10240

template <int RP>
struct Smem {
    // activation and unpacked-weight stages (one group each), groups of nibbles in flight
    static constexpr int kStages = RP <= 64 ? 6 : 4, kRawSlots = RP <= 64 ? 12 : 4;
    static constexpr int kActStage = 128 * 128;  // 128 tokens x 128 B, swizzled
    static constexpr int kBStage = RP * 128;     // int8 weights, swizzled
    static constexpr int kRawSlot = (RP / 8) * 512;  // nibbles of a group: [tile][512]
    static constexpr int kActOff = 0;
    static constexpr int kBOff = kActOff + kStages * kActStage;
    static constexpr int kRawOff = kBOff + kStages * kBStage;
    static constexpr int kWsOff = kRawOff + kRawSlots * kRawSlot;  // fp32 [G][RP]
    static constexpr int kBarOff = kWsOff + kMaxG * RP * 4;
    static constexpr int kTotal = kBarOff + 512 + 1024;  // barriers, + slack to align the base
    static constexpr int kStagePitch = RP / 4 + 4;       // output staging, floats per token
    static_assert(kEpiWarps * 32 * kStagePitch * 4 <= kRawOff, "output staging");
    static_assert(kTotal <= 227 * 1024, "shared memory");
};

// W (eight or four) columns of two blocks: issue, and the wait that makes the registers readable
template <int W>
__device__ __forceinline__ void tmem_issue(uint32_t t0, uint32_t t1, uint32_t (&r)[2][8]) {
    if constexpr (W == 8)
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];"
            : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[0][4]),
              "=r"(r[0][5]), "=r"(r[0][6]), "=r"(r[0][7]), "=r"(r[1][0]), "=r"(r[1][1]),
              "=r"(r[1][2]), "=r"(r[1][3]), "=r"(r[1][4]), "=r"(r[1][5]), "=r"(r[1][6]),
              "=r"(r[1][7])
            : "r"(t0), "r"(t1)
            : "memory");
    else
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%8];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x4.b32 {%4, %5, %6, %7}, [%9];"
            : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[1][0]),
              "=r"(r[1][1]), "=r"(r[1][2]), "=r"(r[1][3])
            : "r"(t0), "r"(t1)
            : "memory");
}
template <int W>
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[2][8]) {
    if constexpr (W == 8)
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0][0]), "+r"(r[0][1]), "+r"(r[0][2]), "+r"(r[0][3]), "+r"(r[0][4]),
                       "+r"(r[0][5]), "+r"(r[0][6]), "+r"(r[0][7]), "+r"(r[1][0]), "+r"(r[1][1]),
                       "+r"(r[1][2]), "+r"(r[1][3]), "+r"(r[1][4]), "+r"(r[1][5]), "+r"(r[1][6]),
                       "+r"(r[1][7])
                     :
                     : "memory");
    else
        asm volatile("tcgen05.wait::ld.sync.aligned;"
                     : "+r"(r[0][0]), "+r"(r[0][1]), "+r"(r[0][2]), "+r"(r[0][3]), "+r"(r[1][0]),
                       "+r"(r[1][1]), "+r"(r[1][2]), "+r"(r[1][3])
                     :
                     : "memory");
}

template <int RP, bool SCL16>
__global__ void __launch_bounds__(kThreads, 1)
gemm_w4a8_tc32_kernel(const GemmArgs a) {
    constexpr int CH = RP / 4;  // columns per epilogue thread
    // A unit is what the MMAs hand to the epilogue: the accumulators of half a group, two blocks
    // of RP columns each.  Two units or four, so one or two groups, fit the tensor memory.
    constexpr int kAccCols = 2 * RP;
    constexpr int kStages = Smem<RP>::kStages, kRawSlots = Smem<RP>::kRawSlots;
    constexpr int kAcc = RP <= 64 ? 4 : 2, kAccGroups = kAcc / 2;
    static_assert(kAcc * kAccCols <= 512, "tensor memory");
    extern __shared__ uint8_t smem_raw[];
    // swizzle atoms need a 1024-byte aligned base
    uint8_t* smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    using S = Smem<RP>;
    const int G = a.groups;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int R = min(a.rows_per_cta, a.n - (int)blockIdx.x * a.rows_per_cta);  // may be ragged
    const int r_tiles = (R + 7) / 8;
    const int tile0 = blockIdx.x * (a.rows_per_cta / 8);
    const int tok0 = blockIdx.y * 128;
    const int m_here = min(128, a.m - tok0);

    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBarOff);
    uint64_t* act_full = bars;                  // [kStages] activations of a group landed
    uint64_t* ab_free = act_full + kStages;     // [kStages] MMAs that read both operands retired
    uint64_t* acc_full = ab_free + kStages;     // [kAcc] unit complete
    // [kFeedWarps][2] epilogue has fetched a half of the group; by group mod kFeedWarps, so that
    // the warp which waits for it sees every phase
    uint64_t* acc_free = acc_full + kAcc;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 2 * kFeedWarps);
    volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

    b2w4_pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&act_full[s], 1);
            mbar_init(&ab_free[s], 1);
        }
        for (int b = 0; b < kAcc; ++b)
            mbar_init(&acc_full[b], 1);
        for (int b = 0; b < 2 * kFeedWarps; ++b)
            mbar_init(&acc_free[b], 4 * ((m_here + 31) / 32));  // the warps that have tokens
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {  // one warp owns the TMEM allocation: 512 columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    auto fail = [&]() {
        *s_abort = 1;
        b2w4_report_timeout(a.status);
    };
    // a wait that looks at the abort word only when the phase is not there yet
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        return mbar_try_wait(bar, parity) || (!*s_abort && mbar_wait(bar, parity));
    };

    if (warp < kEpiWarp0) {
        // ============================ operands and MMAs ==============================
        // Warp w takes every fourth group: when the stage is free it starts the bulk copy of the
        // group's activations and unpacks its nibbles, which it has copied itself, some groups
        // ahead and before the quantiser in front has finished: no barrier between that copy and
        // its use.  Then a lane issues the group's MMAs.  (One warp that issued the MMAs of all
        // groups spent 900 cycles a group on waits that were over and on commits, which set the
        // pace of narrow tiles.  All warps on one group's nibbles at a time, a group took their
        // whole latency; nibbles by one bulk copy per row tile, issuing those took a warp 1700 of
        // a group's 2500 cycles.)
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
        const uint8_t* nib = a.nib + (size_t)tile0 * G * 512 + lane * 16;
        auto fetch = [&](int g) {
            if (g < G) {
                const uint32_t dst =
                    smem_u32(smem + S::kRawOff + (g % kRawSlots) * S::kRawSlot) + lane * 16;
                const uint8_t* src = nib + (size_t)g * 512;
                for (int t = 0; t < r_tiles; ++t)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + t * 512),
                                 "l"(src + (size_t)t * G * 512)
                                 : "memory");
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        constexpr int kOwn = kRawSlots / kFeedWarps;  // groups a warp has in flight
        static_assert(kRawSlots % kFeedWarps == 0, "slots");
        for (int i = 0; i < kOwn; ++i)
            fetch(warp + i * kFeedWarps);
        // only the 8-token atoms that hold real tokens are copied; the MMA reads whatever the
        // rest of the 128-token block holds and the epilogue ignores those rows
        const uint32_t act_bytes = (uint32_t)((m_here + 7) / 8) * 1024;
        b2w4_pdl_wait();  // quantised activations come from the previous kernel
        // chunk `lane` of a tile: 32 k (sub) of weight row `row`; in the operand: atom t (1024 B),
        // row (128 B), 16-byte chunks 2*sub (even k) and 2*sub+1 (odd k), XOR-swizzled with the row
        const int sub = lane >> 3, row = lane & 7;
        const uint32_t even = row * 128 + (((2 * sub) ^ row) << 4);
        const uint32_t odd = row * 128 + (((2 * sub + 1) ^ row) << 4);
        const uint32_t idesc = umma_idesc_i8(RP);
        const uint64_t a_desc0 = umma_desc_k_sw128(smem_u32(smem + S::kActOff));
        const uint64_t b_desc0 = umma_desc_k_sw128(smem_u32(smem + S::kBOff));
        bool ok = true;
        for (int g = warp; g < G; g += kFeedWarps) {
            const int s = g % kStages, round = g / kStages;
            // MMAs left this stage
            if (round > 0 && !__all_sync(0xffffffffu, wait(&ab_free[s], (round - 1) & 1))) {
                ok = false;
                break;
            }
            if (lane == 0) {
                mbar_expect_tx(&act_full[s], act_bytes);
                bulk_g2s(smem + S::kActOff + s * S::kActStage,
                         a.qa + ((size_t)g * a.m_pad + tok0) * 128, act_bytes, &act_full[s]);
            }
            asm volatile("cp.async.wait_group %0;" ::"n"(kOwn - 1) : "memory");
            __syncwarp();
            const uint8_t* raw =
                smem + S::kRawOff + (g % kRawSlots) * S::kRawSlot + lane * 16;
            uint8_t* bst = smem + S::kBOff + s * S::kBStage;
#pragma unroll 4
            for (int t = 0; t < r_tiles; ++t) {
                const uint4 w = *reinterpret_cast<const uint4*>(raw + t * 512);
                // low nibbles = even k, high nibbles = odd k, in two's complement: a nibble in
                // the upper half of a byte is the signed byte 16 q
                constexpr uint32_t kHigh = 0xF0F0F0F0u;
                *reinterpret_cast<uint4*>(bst + t * 1024 + even) =
                    make_uint4((w.x << 4) & kHigh, (w.y << 4) & kHigh, (w.z << 4) & kHigh,
                               (w.w << 4) & kHigh);
                *reinterpret_cast<uint4*>(bst + t * 1024 + odd) =
                    make_uint4(w.x & kHigh, w.y & kHigh, w.z & kHigh, w.w & kHigh);
            }
            fetch(g + kOwn * kFeedWarps);  // a lane reads and refills the same words of the slot
            // make the generic-proxy writes visible to the tensor core's async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                ok = wait(&act_full[s], round & 1);
                // descriptor addresses count 16-byte units
                const uint64_t a_desc = a_desc0 + (uint64_t)(s * (S::kActStage >> 4));
                const uint64_t b_desc = b_desc0 + (uint64_t)(s * (S::kBStage >> 4));
                const int before = g - kAccGroups;  // the group whose sums lay in these units
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int u = g % kAccGroups * 2 + h;
                    ok = ok && (before < 0 || wait(&acc_free[before % kFeedWarps * 2 + h],
                                                   before / kFeedWarps & 1));
                    if (!ok)
                        break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 2; ++j)  // a K = 32 step = a 32-k block
                        umma_i8(tmem_base + (uint32_t)(u * kAccCols + j * RP),
                                a_desc + (uint64_t)((h * 2 + j) * 2),
                                b_desc + (uint64_t)((h * 2 + j) * 2), idesc, 0u);
                    umma_commit(&acc_full[u]);  // the unit's sums are complete
                }
                if (ok)
                    umma_commit(&ab_free[s]);  // both operands' stages may be refilled
            }
            if (!__all_sync(0xffffffffu, ok))
                break;
        }
        if (!ok)
            fail();
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    } else {
        // =============================== epilogue ====================================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpi));
        // the same in all lanes, and the compiler knows: fetch addresses in uniform registers
        const int ew = __shfl_sync(0xffffffffu, warp, 0) - kEpiWarp0;  // 0..15
        const int ch = ew >> 2;                // column quarter
        const int lq = ew & 3;                 // TMEM lane quarter this warp may read
        const int tok = tok0 + lq * 32 + lane;
        // a warp whose 32 tokens all lie past the last row has no chain to run
        const bool active = lq * 32 < m_here;
        // weight scales / 16 -> fp32 [G][RP] (column = row of the CTA), shared by all tokens
        {
            float* wsf = reinterpret_cast<float*>(smem + S::kWsOff);
            // eight scales of one (tile, group) are contiguous
            for (int i = ew * 32 + lane; i < G * (RP / 8); i += kEpiWarps * 32) {
                const int t = i / G, g = i - t * G;
                float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
                if (t < r_tiles) {
                    const size_t idx = ((size_t)(tile0 + t) * G + g) * 8;
                    if (SCL16) {
                        const uint4 raw = *reinterpret_cast<const uint4*>(
                            reinterpret_cast<const __half*>(a.scl) + idx);
                        const __half2* h = reinterpret_cast<const __half2*>(&raw);
                        const float2 f0 = __half22float2(h[0]), f1 = __half22float2(h[1]);
                        const float2 f2 = __half22float2(h[2]), f3 = __half22float2(h[3]);
                        lo = make_float4(f0.x, f0.y, f1.x, f1.y);
                        hi = make_float4(f2.x, f2.y, f3.x, f3.y);
                    } else {
                        const float4* f = reinterpret_cast<const float4*>(
                            reinterpret_cast<const float*>(a.scl) + idx);
                        lo = f[0];
                        hi = f[1];
                    }
                }
                auto scaled = [](float4 v) {
                    return make_float4(__fmul_rn(v.x, 0.0625f), __fmul_rn(v.y, 0.0625f),
                                       __fmul_rn(v.z, 0.0625f), __fmul_rn(v.w, 0.0625f));
                };
                *reinterpret_cast<float4*>(wsf + g * RP + t * 8) = scaled(lo);
                *reinterpret_cast<float4*>(wsf + g * RP + t * 8 + 4) = scaled(hi);
            }
        }
        // named barrier among the epilogue warps only
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps * 32) : "memory");
        b2w4_pdl_wait();  // the quantiser's scales; and y may still be in use before this
        const float* wsf = reinterpret_cast<const float*>(smem + S::kWsOff) + ch * CH;
        const bool has_tok = tok < a.m;
        // the token's four block scales of a group are one 16-byte load, fetched two groups
        // ahead (a group's chain is long enough to cover the load)
        const float4* as4 = reinterpret_cast<const float4*>(a.as) + tok;
        auto load_as = [&](int g) {
            return (has_tok && g < G) ? as4[(size_t)g * a.m_pad]
                                      : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        float4 a0 = load_as(0), a1 = load_as(1);
        uint64_t acc2[CH / 2];  // the chain values, columns (2i, 2i + 1) side by side
#pragma unroll
        for (int i = 0; i < CH / 2; ++i)
            acc2[i] = 0ull;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(lq * 32) << 16) + (uint32_t)(ch * CH);
        bool live = true;
        if (active) {
            auto unit_wait = [&](uint64_t* full, int parity) {
                const bool ready = mbar_try_wait(full, parity);
                if (!__all_sync(0xffffffffu, ready))
                    live &= __all_sync(0xffffffffu, ready || wait(full, parity)) != 0;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            };
            auto unit_done = [&](uint64_t* free) {  // every fetch of the unit is in registers
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(free);
            };
            // A chunk is eight columns (the last one of a thread may be four) of two blocks.
            constexpr int kHalf = (CH + 7) / 8, kChunks = 2 * kHalf;  // per block pair, per group
            static_assert(CH % 4 == 0, "columns");
            auto group = [&](int g, float4& scales) {
                const float asv[4] = {scales.x, scales.y, scales.z, scales.w};
                scales = load_as(g + 2);
                const float* ws = wsf + g * RP;
                const int u = g % kAccGroups * 2, parity = g / kAccGroups & 1;
                uint64_t* free = acc_free + g % kFeedWarps * 2;
                auto step = [&](auto chunk) {
                    constexpr int i = decltype(chunk)::value;
                    constexpr int j = i / kHalf * 2, c = i % kHalf * 8, W = c + 8 <= CH ? 8 : 4;
                    constexpr int h = j / 2;  // half of the group
                    if constexpr (c == 0)
                        unit_wait(&acc_full[u + h], parity);
                    uint32_t r[2][8];
                    const uint32_t t = lane_addr + (uint32_t)((u + h) * kAccCols + c);
                    tmem_issue<W>(t, t + RP, r);
                    tmem_wait<W>(r);
                    if constexpr (i + 1 == kChunks || i + 1 == kHalf)
                        unit_done(free + h);
                    // two blocks, in ascending order
                    const uint64_t s0 = b2w4_pack2(asv[j], asv[j]);
                    const uint64_t s1 = b2w4_pack2(asv[j + 1], asv[j + 1]);
#pragma unroll
                    for (int e4 = 0; e4 < W; e4 += 4) {
                        const ulonglong2 w2 = *reinterpret_cast<const ulonglong2*>(ws + c + e4);
                        auto sums = [&](int b, int e) {
                            return b2w4_pack2(__int2float_rn((int)r[b][e]),
                                              __int2float_rn((int)r[b][e + 1]));
                        };
                        uint64_t& lo = acc2[(c + e4) / 2];
                        uint64_t& hi = acc2[(c + e4) / 2 + 1];
                        lo = b2w4_fma2(sums(0, e4), b2w4_mul2(w2.x, s0), lo);
                        hi = b2w4_fma2(sums(0, e4 + 2), b2w4_mul2(w2.y, s0), hi);
                        lo = b2w4_fma2(sums(1, e4), b2w4_mul2(w2.x, s1), lo);
                        hi = b2w4_fma2(sums(1, e4 + 2), b2w4_mul2(w2.y, s1), hi);
                    }
                };
                [&]<int... I>(std::integer_sequence<int, I...>) {
                    (step(std::integral_constant<int, I>()), ...);
                }(std::make_integer_sequence<int, kChunks>());
            };
            // Two groups a turn need no moves of the scales, but the code is twice as long: taken where
            // a group's is short.  Time of two a turn to one, K = 1024 / 2560 / 9728, one to five sizes
            // each, fp16 and fp32 scales alike: 32 columns 0.99 / 0.98 / 0.97, 48 1.00 / 0.99 / 0.98, 64
            // 0.98 / 0.97 / 0.96, 80 0.98 / 0.96 / 0.95, 96 1.02 / 1.01 / 1.00, 112 1.02 / 1.01 / 1.01,
            // 128 1.01 / 1.01 / 1.01.
            constexpr bool kPairs = RP <= 80;
            for (int g = 0; g < G; g += kPairs ? 2 : 1) {
                group(g, a0);
                if constexpr (!kPairs) {
                    const float4 t = a0;  // of the group after the next
                    a0 = a1;
                    a1 = t;
                } else if (g + 1 < G) {
                    group(g + 1, a1);
                }
            }
        }
        if (!live)
            fail();
        // Output: a thread holds one token's CH columns, which lie CH*4 bytes apart from the
        // next token's in y.  Stage the warp's 32 x CH block in shared memory (the operand
        // ring is idle: the last accumulator was complete, so every MMA and copy has
        // retired) and store token rows with the lanes running along the columns.
        if (active && live && !*s_abort) {
            constexpr int SP = S::kStagePitch;  // 16-byte aligned rows
            float* stage = reinterpret_cast<float*>(smem + S::kActOff) + ew * (32 * SP);
            const int n0 = blockIdx.x * a.rows_per_cta + ch * CH;
#pragma unroll
            for (int c = 0; c < CH; c += 4) {
                float4 v;
                b2w4_unpack2(acc2[c / 2], v.x, v.y);
                b2w4_unpack2(acc2[c / 2 + 1], v.z, v.w);
                if (a.activation != B2W4_NONE) {
                    float* e = &v.x;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (b2w4_act_applies(n0 + c + i, a.activation, a.act_n_begin,
                                             a.act_n_len, a.n))
                            e[i] = gemm_activation(e[i], a.activation);
                }
                *reinterpret_cast<float4*>(stage + lane * SP + c) = v;
            }
            __syncwarp();
            const int tok_w = tok0 + lq * 32;  // first token of this warp
            const int rows_w = min(32, a.m - tok_w);
            const bool vec_ok = (a.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(a.y) & 15) == 0;
            constexpr int V = CH / 4;  // float4s per token row
#pragma unroll 4
            for (int i = lane; i < rows_w * V; i += 32) {
                const int rr = i / V, c = (i - rr * V) * 4;
                const float4 v = *reinterpret_cast<const float4*>(stage + rr * SP + c);
                float* dst = a.y + (size_t)(tok_w + rr) * a.ldc + n0 + c;
                const int left = R - (ch * CH + c);  // valid columns from here on
                if (left >= 4 && vec_ok) {
                    *reinterpret_cast<float4*>(dst) = v;
                } else {
                    if (left > 0) dst[0] = v.x;
                    if (left > 1) dst[1] = v.y;
                    if (left > 2) dst[2] = v.z;
                    if (left > 3) dst[3] = v.w;
                }
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem_base), "r"(512)
                     : "memory");
    }
}

template <int RP>
int launch_rp(b2w4_ctx* ctx, const GemmArgs& a, bool scl16, dim3 grid) {
    using S = Smem<RP>;
    auto kern = scl16 ? gemm_w4a8_tc32_kernel<RP, true> : gemm_w4a8_tc32_kernel<RP, false>;
    static b2w4_smem_optin configured[2];  // per instantiation and device
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, S::kTotal, configured[scl16]));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, grid, dim3(kThreads), S::kTotal,
                                       ctx->stream, a));
    ctx->launches++;
    return B2W4_OK;
}

// What a group costs beside its columns, in columns.
constexpr int kFixedColumns = 24;
// accumulator columns of the instantiation that takes r row tiles
int columns_for(int r) { return r <= 4 ? 32 : (r + 1) / 2 * 16; }

// Rows per CTA.  The fp32 chain paces a CTA, so its time grows with the accumulator columns
// of its instantiation (plus a fixed part per group); the launch takes as many rounds as the
// CTAs need on the SMs.  Pick the tile count with the least product.
int row_tiles(int tiles, int token_blocks, int sm_count) {
    int best = 1;
    long best_cost = -1;
    for (int r = 1; r <= 16; ++r) {
        const long ctas = (long)((tiles + r - 1) / r) * token_blocks;
        const long rounds = (ctas + sm_count - 1) / sm_count;
        const long cost = rounds * (columns_for(r) + kFixedColumns);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = r;
        }
    }
    return best;
}

}  // namespace

// Quantises the activations per 32 values (separate launch), then runs the kernel above.
int b2w4_launch_gemm_tc32(b2w4_ctx* ctx, const b2w4_weight* w, const float* x, int lda, float* y,
                          int ldc, int m, int activation, int act_n_begin, int act_n_len,
                          const b2w4_rows* from) {
    const int G = w->groups;
    if (G > kMaxG)
        return b2w4_fail(ctx, B2W4_E_INVALID, "gemm: K=%d exceeds the scale staging (K<=10240)",
                         w->k);
    const int m_pad = (m + 127) / 128 * 128;
    void *qa = nullptr, *as = nullptr;
    int rc;
    if ((rc = b2w4_reserve(ctx, SCR_QA, (size_t)G * m_pad * 128, &qa)) != B2W4_OK ||
        (rc = b2w4_reserve(ctx, SCR_AS, sizeof(float) * (size_t)G * m_pad * 4, &as)) != B2W4_OK)
        return rc;
    if ((rc = b2w4_launch_quantize_umma(ctx, x, lda, m, w->k, m_pad, B2W4_ACT_G32,
                                        static_cast<int8_t*>(qa), static_cast<float*>(as),
                                        from)) !=
        B2W4_OK)
        return rc;
    const int token_blocks = m_pad / 128;
    const int r_tiles = row_tiles(w->tiles, token_blocks, ctx->sm_count);
    GemmArgs a;
    a.nib = reinterpret_cast<const uint8_t*>(w->nib);
    a.scl = w->scl;
    a.qa = static_cast<const int8_t*>(qa);
    a.as = static_cast<const float*>(as);
    a.y = y;
    a.status = ctx->status_dev;
    a.ldc = ldc;
    a.m = m;
    a.m_pad = m_pad;
    a.n = w->n;
    a.groups = G;
    a.tiles = w->tiles;
    a.rows_per_cta = r_tiles * 8;
    a.activation = activation;
    a.act_n_begin = act_n_begin;
    a.act_n_len = act_n_len;
    const dim3 grid((w->tiles + r_tiles - 1) / r_tiles, token_blocks);
    const bool scl16 = w->scales_fp16 != 0;
    switch (columns_for(r_tiles)) {
    case 32: return launch_rp<32>(ctx, a, scl16, grid);
    case 48: return launch_rp<48>(ctx, a, scl16, grid);
    case 64: return launch_rp<64>(ctx, a, scl16, grid);
    case 80: return launch_rp<80>(ctx, a, scl16, grid);
    case 96: return launch_rp<96>(ctx, a, scl16, grid);
    case 112: return launch_rp<112>(ctx, a, scl16, grid);
    default: return launch_rp<128>(ctx, a, scl16, grid);
    }
}
