// Causal attention of a long run of tokens over the cache on tcgen05.mma kind::f16: the products
// of attention_tile.cuh with every fp32 operand as the sum of three bf16 numbers.
//
// x = h + m + l, each the bf16 nearest to what is left: 24 bits, so the sum is x unless x has bits
// below 2^-133, the smallest bf16, or rounds to infinity.  A product takes six of the nine piece products, the small ones first,
//   l h' + h l' + m m' + m h' + h m' + h h'
// what is left out is below 2^-24 of |x x'|; sums are fp32 in tensor memory.  Scores,
// probabilities (exp in 64 bits, rounded once), maxima and sums stay fp32, and the output's sum
// over key blocks is kept in registers with one rounding per block.
//
// A block takes 128 (token, head) rows of one kv head against blocks of 64 keys, and is alone on
// its multiprocessor: the pieces of two blocks of keys and values fill shared memory.  The MMA's A
// operands (Q's h and m, the probabilities' pieces) are in tensor memory.  A score has two sums,
// which the softmax adds: an MMA of 128 rows takes 47 cycles for 64 columns and 66 for 128
// (measured), so Q's m meets the keys' h and m side by side, as 128 columns.  Roles:
//   rows       eight warps, two threads to a row: 32 of the 64 scores each (running maximum, exp in
//              64 bits, pieces of the probabilities back to tensor memory) and DIM / 2 of the
//              output's sums, o = o * alpha + P V of the block
//   MMA        a thread for the scores, a block ahead, and one for P V
//   split      seven warps for the keys, seven for the values: from global memory to pieces in the
//              MMA's layout (values transposed)
// A score's h h' products go to one sum for one half of the features and to the other for the
// other: a sum in tensor memory truncates, by less the smaller it is.
// What bounds it: a step of 64 keys takes about 7700 cycles at DIM = 128.  Its MMAs alone take 2050
// (scores) and 1600 (P V), its softmax and splits about 4000 of each scheduler (conversions and
// logic at half rate, paired fp32 instructions two to three cycles each); the exp lengthens the rows'
// chain by 1500 (530 instructions of a scheduler's 64-bit pipe, which is busy for 1100); shared
// memory serves MMAs, splits and loads for about 3000.
// Measured against the tile form: attn_tensor (decoder_ops.cu).  Tried with an exp in 32 bits, 1500
// tokens of 32 / 8 heads of 128 (167 us; 208 with this one, 214 with the checks below): all products
// with m and h of the keys side by side 156 (error 2.3e-7 instead of 1.8e-7), each alone 188; three
// warps each to split 197, five 170.
// Some tiles go to the fp32 form (attention_tile.cuh), which has the rule for values of probability
// zero; nothing is written before that is known:
//   a result that is not finite, or not zero and below 2^-100 (a product of pieces may have been lost)
//   a query, key or value that its pieces do not sum to (what is left after the third is not zero)
//   a probability that its pieces do not sum to (below 2^-110, at most 2^-134 is lost), where a
//   value is 2^32 or more, or a result zero or below 2^-60: up to 2^17 keys lose less than 2^-85
// Every wait is bounded; on a timeout the kernel flags the status word and drains.
#include "attention_tile.cuh"
#include "tcgen05_ops.cuh"

namespace {

constexpr int kKeys = 64;    // keys of a step
constexpr int kRows = 128;   // (token, head) rows of a block
constexpr int kRowWarps = 8, kScoreWarp = 8, kOutWarp = 9, kSplitWarp0 = 10;
constexpr int kSplitWarps = 7;  // for the keys, and as many for the values
constexpr int kTcThreads = (kSplitWarp0 + 2 * kSplitWarps) * 32;
constexpr float kLarge = 0x1p32f, kSmall = 0x1p-100f, kSmallLost = 0x1p-60f;  // see above
constexpr int kRegsStart = 80, kRegsRows = 128, kRegsOther = 56;
static_assert(kRowWarps * 32 == kAttnThreads);
static_assert(2 * kRegsRows + 4 * kRegsOther <= 6 * kRegsStart, "registers of the block");

template <int DIM>
struct TcSmem {
    // A bf16 piece of a block of values: DIM rows of 64 keys, 128 bytes each; of 64 features of a
    // block of keys: 64 rows.  Keys lie as [64 features][piece], so that h and m are neighbours.
    static constexpr int kValuePiece = DIM * 128, kKeyPiece = kKeys * 128;
    static constexpr int kBuf = 3 * kKeys * DIM * 2;
    static constexpr int kK = 0, kV = 2 * kBuf;
    static constexpr int kQ = 4 * kBuf;  // Q's smallest piece: [64 features][128 rows]
    static constexpr int kQPart = kRows * 128;
    static constexpr int kMax = kQ + kRows * DIM * 2;      // float [2 parities][2 halves][kRows]
    static constexpr int kBar = kMax + 4 * kRows * 4;
    static constexpr int kTotal = kBar + 256;
    static_assert(TileSmem<DIM, 64>::kBytes <= kMax, "the fp32 form's buffers");
    static_assert(kTotal <= 227 * 1024, "shared memory");
};
// tensor memory, columns: Q's pieces h and m, two sums of the scores, the probabilities' pieces,
// P V
template <int DIM>
struct TcTmem {
    static constexpr int kQ = 0, kS = DIM, kP = kS + 2 * kKeys, kO = kP + 3 * kKeys / 2;
    static_assert(kO + DIM <= 512, "tensor memory");
};

// kind::f16, bf16 operands, fp32 accumulate, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}
// A from tensor memory, B from shared memory
__device__ __forceinline__ void umma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
#define B2W4_R8(r, o) "r"(r[o]), "r"(r[o + 1]), "r"(r[o + 2]), "r"(r[o + 3]), "r"(r[o + 4]), \
                      "r"(r[o + 5]), "r"(r[o + 6]), "r"(r[o + 7])
#define B2W4_W8(r, o) "=r"(r[o]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]),            \
                      "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
// A from shared memory too
__device__ __forceinline__ void umma_bf16_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                             uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 16 columns of the thread's row: issue, and the wait that makes them readable
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, "
        "%11, %12, %13, %14, %15}, [%16];"
        : B2W4_W8(r, 0), B2W4_W8(r, 8)
        : "r"(taddr)
        : "memory");
}
#define B2W4_RW8(r, o) "+r"(r[o]), "+r"(r[o + 1]), "+r"(r[o + 2]), "+r"(r[o + 3]),           \
                       "+r"(r[o + 4]), "+r"(r[o + 5]), "+r"(r[o + 6]), "+r"(r[o + 7])
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[16], uint32_t (&b)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : B2W4_RW8(a, 0), B2W4_RW8(a, 8), B2W4_RW8(b, 0), B2W4_RW8(b, 8)
                 :
                 : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, "
        "%10, %11, %12, %13, %14, %15};" ::B2W4_R8(r, 0),
        B2W4_R8(r, 8), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() {
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// The next piece of two numbers, low half = lo; they keep what is left (exact).
__device__ __forceinline__ uint32_t take_piece(uint64_t& v) {
    float lo, hi;
    b2w4_unpack2(v, lo, hi);
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(hi), "f"(lo));
    v = b2w4_sub2(v, b2w4_pack2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)));
    return p;
}

// exp of x <= 0 (NaN stays), in 64 bits and rounded once.  After Tang, Table-driven implementation of
// the exponential function (1989): x = i ln 2 / 32 + r, 2^(i % 32 / 32) from lane i % 32 (a whole
// warp calls this), the Taylor series of e^r - 1 to r^5 with its last term economised (Chebyshev):
// relative error below 2^-43, so about three results in a million are rounded to the neighbour of
// the nearest number.  No branch, eight instructions of the 64-bit pipe and two conversions: 1500
// tokens of 32 / 8 heads of 128 take 208 us, with CUDA's exp 264, without a table 223.
__device__ __forceinline__ float exp_neg(float x, double lane_power) {
    constexpr double kStep = 0.02166084939249829;  // ln 2 / 32
    constexpr double kMagic = 6755399441055744.;   // 1.5 * 2^52: the sum's low bits are the integer
    const double xd = (double)(x < -110.f ? -110.f : x);  // exp(-104) is zero in 32 bits
    const double t = fma(xd, 1. / kStep, kMagic);
    const double r = fma(t - kMagic, -kStep, xd);  // |r| <= kStep / 2
    const int i = __double2loint(t);
    const int hi = __shfl_sync(0xffffffffu, __double2hiint(lane_power), i & 31);
    const int lo = __shfl_sync(0xffffffffu, __double2loint(lane_power), i & 31);
    const double power = __hiloint2double(hi + ((i >> 5) << 20), lo);
    constexpr double a = kStep / 2;  // r^5 / 120 as a cubic
    double p = fma(r, 1. / 24., 1. / 6. + a * a * (5. / 480.));
    p = fma(p, r, 0.5);
    p = fma(p, r, 1. - a * a * a * a * (1. / 384.));
    return (float)fma(power, p * r, power);
}

// kAttnThreads threads of the larger block
struct PartSync {
    static __device__ __forceinline__ void sync() {
        asm volatile("bar.sync 2, %0;" ::"n"(kAttnThreads) : "memory");
    }
    static __device__ __forceinline__ bool any(bool v) {
        int r;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.ne.s32 p, %1, 0;\n\t"
            "barrier.cta.red.or.pred q, 2, %2, p;\n\t"
            "selp.s32 %0, 1, 0, q;\n\t}"
            : "=r"(r)
            : "r"((int)v), "n"(kAttnThreads)
            : "memory");
        return r != 0;
    }
};

template <int DIM>
__global__ void __launch_bounds__(kTcThreads, 1)
attention_tc_kernel(const float* __restrict__ q, const float* __restrict__ k_cache,
                    const float* __restrict__ v_cache, float* __restrict__ out, int tokens,
                    int heads, int kv_heads, int past0, const int* __restrict__ past_dev,
                    int capacity, float scale, int tq, int* status) {
    using S = TcSmem<DIM>;
    using T = TcTmem<DIM>;
    extern __shared__ __align__(1024) uint8_t smem[];  // swizzle atoms: 1024-byte aligned
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kBar);
    uint64_t* q_full = bars;            // Q's pieces in tensor memory
    uint64_t* s_full = bars + 1;        // scores of a block complete
    uint64_t* s_free = bars + 2;        // ... and in registers
    uint64_t* p_full = bars + 3;        // probabilities' pieces in tensor memory
    uint64_t* o_full = bars + 4;        // P V of a block complete (and P read)
    uint64_t* o_free = bars + 5;        // ... and in registers
    uint64_t* drained = bars + 6;       // [2] every MMA retired
    uint64_t* k_full = bars + 8;        // [2] pieces of a block
    uint64_t* k_free = bars + 10;       // [2]
    uint64_t* v_full = bars + 12;       // [2]
    uint64_t* v_free = bars + 14;       // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* s_abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_odd = s_abort + 1;   // to the fp32 form
    volatile int* s_lost = s_abort + 2;  // bits of a probability
    float* s_max = reinterpret_cast<float*>(smem + S::kMax);

    b2w4_pdl_launch_dependents();
    if (threadIdx.x == 0) {
        mbar_init(q_full, kRowWarps);
        mbar_init(s_full, 1);
        mbar_init(s_free, kRowWarps);
        mbar_init(p_full, kRowWarps);
        mbar_init(o_full, 1);
        mbar_init(o_free, kRowWarps);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&drained[b], 1);
            mbar_init(&k_full[b], kSplitWarps);
            mbar_init(&k_free[b], 1);
            mbar_init(&v_full[b], kSplitWarps);
            mbar_init(&v_free[b], 1);
        }
        *s_abort = 0;
        *s_odd = *s_lost = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kScoreWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(tmem_slot)), "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    auto fail = [&]() {
        *s_abort = 1;
        b2w4_report_timeout(status);
    };
    // a wait that looks at the abort word only when the phase is not there yet
    auto wait = [&](uint64_t* bar, uint32_t parity) {
        return mbar_try_wait(bar, parity) || (!*s_abort && mbar_wait(bar, parity));
    };
    auto warp_wait = [&](uint64_t* bar, uint32_t parity) {
        return __all_sync(0xffffffffu, wait(bar, parity)) != 0;
    };
    auto warp_arrive = [&](uint64_t* bar) {
        __syncwarp();
        if (lane == 0)
            mbar_arrive(bar);
    };

    b2w4_pdl_wait();
    const int past = past_dev ? min(*past_dev, capacity - tokens) : past0;
    const int rep = heads / kv_heads;
    // the last tiles see the most keys: they go first, of all kv heads
    const int kvh = blockIdx.x, t0 = (int)(gridDim.y - 1 - blockIdx.y) * tq;
    const int vis_max = past + min(t0 + tq, tokens);  // keys the tile's last token sees
    const int steps = (vis_max + kKeys - 1) / kKeys;
    const float* kc = k_cache + (size_t)kvh * capacity * DIM;
    const float* vc = v_cache + (size_t)kvh * capacity * DIM;
    // row r of the tile: token t0 + r / rep, head kvh * rep + r % rep; rows past the tile's
    // tokens see no key
    auto row_visible = [&](int r) {
        return (r < tq * rep && t0 + r / rep < tokens) ? past + t0 + r / rep + 1 : 0;
    };
    auto row_offset = [&](int r) {
        return ((size_t)(t0 + r / rep) * heads + kvh * rep + r % rep) * DIM;
    };

    // row, chunk of 16 bytes -> bytes in 128-byte rows: 8-row atoms, chunks swizzled with the row
    auto place = [](int row, int chunk) {
        return (uint32_t)((row >> 3) * 1024 + (row & 7) * 128 + ((chunk ^ (row & 7)) << 4));
    };

    if (warp < kRowWarps) {
        // ================================== rows =====================================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsRows));
        const int quarter = warp & 3, half = warp >> 2;  // of the tensor memory's lanes; of columns
        const int row = quarter * 32 + lane;
        const int vis = row_visible(row);
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        // both threads of a quarter's rows have come here
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(3 + quarter) : "memory"); };
        {
            const float4* src = reinterpret_cast<const float4*>(q + (vis ? row_offset(row) : 0));
            uint64_t left = 0ull;
#pragma unroll 1
            for (int c = half * (DIM / 2); c < (half + 1) * (DIM / 2); c += 32) {
                uint64_t v[16];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 f = vis ? src[c / 4 + i] : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[2 * i] = b2w4_pack2(f.x, f.y);
                    v[2 * i + 1] = b2w4_pack2(f.z, f.w);
                }
                uint32_t r[16];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        r[i] = take_piece(v[i]);
                    if (p < 2)
                        tmem_st16(lane_addr + T::kQ + p * (DIM / 2) + c / 2, r);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    left |= v[i];
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    *reinterpret_cast<uint4*>(smem + S::kQ + c / 64 * S::kQPart +
                                              place(row, c % 64 / 8 + i)) =
                        make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
            }
            if (left)
                *s_odd = 1;
            tmem_st_wait();
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            warp_arrive(q_full);
        }
        const double lane_power = exp2(lane / 32.);
        float m = -INFINITY, l = 0.f, alpha = 1.f;  // alpha: of the block before
        constexpr int kOwn = DIM / 2;               // the thread's share of the output
        uint64_t acc[kOwn / 2];
#pragma unroll
        for (int i = 0; i < kOwn / 2; ++i)
            acc[i] = 0ull;
        // No way out of the loop: the two threads of a row meet at a barrier once a step.
        bool live = true;
        auto await = [&](uint64_t* bar, uint32_t parity) {
            if (live && !warp_wait(bar, parity)) {
                live = false;
                fail();
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        };
        // the thread's share of P V of block j, whose factor is `alpha`
        auto take_output = [&]() {
            const uint64_t al = b2w4_pack2(alpha, alpha);
#pragma unroll
            for (int c = 0; c < kOwn; c += 32) {
                uint32_t r0[16], r1[16];
                tmem_ld16(lane_addr + T::kO + half * kOwn + c, r0);
                tmem_ld16(lane_addr + T::kO + half * kOwn + c + 16, r1);
                tmem_ld_wait(r0, r1);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const uint32_t* r = i < 8 ? r0 : r1;
                    acc[c / 2 + i] = b2w4_fma2(acc[c / 2 + i], al,
                                               b2w4_pack2(__uint_as_float(r[2 * (i & 7)]),
                                                          __uint_as_float(r[2 * (i & 7) + 1])));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            warp_arrive(o_free);
        };
        for (int j = 0; j < steps; ++j) {
            await(s_full, j & 1);
            uint64_t s[16];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t a[16], b[16];
                tmem_ld16(lane_addr + T::kS + half * 32 + 16 * h, a);
                tmem_ld16(lane_addr + T::kS + kKeys + half * 32 + 16 * h, b);
                tmem_ld_wait(a, b);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    s[8 * h + i] = b2w4_mul2(
                        add2(b2w4_pack2(__uint_as_float(a[2 * i]), __uint_as_float(a[2 * i + 1])),
                             b2w4_pack2(__uint_as_float(b[2 * i]), __uint_as_float(b[2 * i + 1]))),
                        b2w4_pack2(scale, scale));
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            warp_arrive(s_free);
            const int seen = vis - j * kKeys - half * 32;  // of the thread's keys, the row sees
            if (seen < 32) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float a, b;
                    b2w4_unpack2(s[i], a, b);
                    s[i] = b2w4_pack2(2 * i < seen ? a : -INFINITY,
                                      2 * i + 1 < seen ? b : -INFINITY);
                }
            }
            float top = m;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float a, b;
                b2w4_unpack2(s[i], a, b);
                top = fmaxf(fmaxf(top, a), b);
            }
            float* mx = s_max + (j & 1) * 2 * kRows;
            mx[half * kRows + row] = top;
            pair_sync();
            top = fmaxf(top, mx[(1 - half) * kRows + row]);
            const float base = top == -INFINITY ? 0.f : top;  // nothing seen yet: all terms zero
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float a, b;
                b2w4_unpack2(s[i], a, b);
                s[i] = b2w4_pack2(exp_neg(__fsub_rn(a, base), lane_power),
                                  exp_neg(__fsub_rn(b, base), lane_power));
            }
            uint64_t sum[4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                sum[i] = add2(add2(s[i], s[i + 4]), add2(s[i + 8], s[i + 12]));
            sum[0] = add2(add2(sum[0], sum[1]), add2(sum[2], sum[3]));
            float sum0, sum1;
            b2w4_unpack2(sum[0], sum0, sum1);
            const float factor = exp_neg(__fsub_rn(m, base), lane_power);
            m = top;
            l = __fadd_rn(__fmul_rn(l, factor), __fadd_rn(sum0, sum1));
            uint32_t pieces[3][16];
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    pieces[p][i] = take_piece(s[i]);
            uint64_t left = 0ull;
#pragma unroll
            for (int i = 0; i < 16; ++i)
                left |= s[i];
            if (left)
                *s_lost = 1;
            // the product before has read the probabilities
            if (j)
                await(o_full, (j - 1) & 1);
#pragma unroll
            for (int p = 0; p < 3; ++p)
                tmem_st16(lane_addr + T::kP + p * (kKeys / 2) + half * 16, pieces[p]);
            tmem_st_wait();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            warp_arrive(p_full);
            if (j)
                take_output();
            alpha = factor;
        }
        await(o_full, (steps - 1) & 1);
        take_output();
        // the other thread's part of the sum (the other parity's words: they may still be read)
        float* mx = s_max + (steps & 1) * 2 * kRows;
        mx[half * kRows + row] = l;
        pair_sync();
        const float total = __fadd_rn(mx[row], mx[kRows + row]);
        // every warp's words are there since the last block's probabilities were
        const bool lost = *s_lost;
        const float small = lost ? kSmallLost : kSmall;
        bool odd = false;
        if (lost)
            for (int i = threadIdx.x; i < vis_max * (DIM / 4); i += kAttnThreads) {
                const float4 f = reinterpret_cast<const float4*>(vc)[i];
                odd |= fmaxf(fmaxf(fabsf(f.x), fabsf(f.y)), fmaxf(fabsf(f.z), fabsf(f.w))) >= kLarge;
            }
#pragma unroll
        for (int i = 0; i < kOwn / 2; ++i) {
            float a, b;
            b2w4_unpack2(acc[i], a, b);
            a = __fdiv_rn(a, total);
            b = __fdiv_rn(b, total);
            auto plain = [&](float v) {
                return (v == 0.f && !lost) || (fabsf(v) >= small && fabsf(v) < INFINITY);
            };
            odd |= vis && (!plain(a) || !plain(b));
            acc[i] = b2w4_pack2(a, b);
        }
        // One answer for all rows, as the fp32 form has barriers that each of them must meet: the MMA
        // threads still wait for their last commits and may report a failure at any time.
        const bool failed = PartSync::any(*s_abort);
        const bool again = PartSync::any(odd || *s_odd);
        if (vis && !again && !failed) {
            ulonglong2* dst = reinterpret_cast<ulonglong2*>(out + row_offset(row) + half * kOwn);
#pragma unroll
            for (int i = 0; i < kOwn / 4; ++i)
                dst[i] = make_ulonglong2(acc[2 * i], acc[2 * i + 1]);
        }
        // the last product has retired, so nothing reads or writes the buffers any more
        if (again && !failed) {
            const int tq_part = 64 / rep, end = min(tokens, t0 + tq);
            for (int t = t0; t < end; t += tq_part) {
                attention_tile<DIM, 64, true, PartSync>(
                    q, k_cache, v_cache, out, min(end, t + tq_part), heads, kv_heads, past,
                    capacity, scale, tq_part, kvh, t, reinterpret_cast<float*>(smem));
                PartSync::sync();  // the buffers are free again
            }
        }
    } else {
      asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
      if (warp == kScoreWarp) {
        // ============================ MMA issue: scores ==============================
        if (lane == 0) {
            const uint64_t k_desc0 = umma_desc_k_sw128(smem_u32(smem + S::kK));
            const uint64_t q_desc = umma_desc_k_sw128(smem_u32(smem + S::kQ));
            bool ok = wait(q_full, 0);
            for (int j = 0; j < steps && ok; ++j) {
                ok = wait(&k_full[j & 1], (j >> 1) & 1) && (j == 0 || wait(s_free, (j - 1) & 1));
                if (!ok)
                    break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t d = k_desc0 + (uint64_t)((j & 1) * (S::kBuf >> 4));
                // features 16 k of piece p of the keys; h and m are the pieces 0 and 1
                auto keys = [&](int k, int p) {
                    return d + (uint64_t)(((k / 4 * 3 + p) * S::kKeyPiece + k % 4 * 32) >> 4);
                };
                constexpr uint32_t one = umma_idesc_bf16(kKeys), two = umma_idesc_bf16(2 * kKeys);
                const uint32_t qh = tmem + T::kQ, qm = qh + DIM / 2;
                const uint32_t s0 = tmem + T::kS, s1 = s0 + kKeys;
                // the smallest products first: l h' and h l', m h' and m m', h m', then h h' of
                // one half of the features and of the other
#pragma unroll
                for (int k = 0; k < DIM / 16; ++k) {
                    umma_bf16_ss(s0, q_desc + (uint64_t)((k / 4 * S::kQPart + k % 4 * 32) >> 4),
                                 keys(k, 0), one, k > 0);
                    umma_bf16_ts(s1, qh + k * 8, keys(k, 2), one, k > 0);
                }
#pragma unroll
                for (int k = 0; k < DIM / 16; ++k)
                    umma_bf16_ts(s0, qm + k * 8, keys(k, 0), two, 1u);
#pragma unroll
                for (int k = 0; k < DIM / 16; ++k)
                    umma_bf16_ts(k % 2 ? s1 : s0, qh + k * 8, keys(k, 1), one, 1u);
#pragma unroll
                for (int k = 0; k < DIM / 16; ++k)
                    umma_bf16_ts(k < DIM / 32 ? s0 : s1, qh + k * 8, keys(k, 0), one, 1u);
                umma_commit(s_full);
                umma_commit(&k_free[j & 1]);
            }
            if (!ok)
                fail();
            umma_commit(&drained[0]);
            if (!mbar_wait(&drained[0], 0))
                fail();
        }
      } else if (warp == kOutWarp) {
        // ============================== MMA issue: P V ===============================
        if (lane == 0) {
            const uint64_t v_desc0 = umma_desc_k_sw128(smem_u32(smem + S::kV));
            // pieces of P and V, the smallest products first
            constexpr int kPa[6] = {2, 0, 1, 1, 0, 0}, kPb[6] = {0, 2, 1, 0, 1, 0};
            bool ok = true;
            for (int j = 0; j < steps; ++j) {
                ok = wait(&v_full[j & 1], (j >> 1) & 1) &&
                     (j == 0 || wait(o_free, (j - 1) & 1)) && wait(p_full, j & 1);
                if (!ok)
                    break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t d = v_desc0 + (uint64_t)((j & 1) * (S::kBuf >> 4));
#pragma unroll
                for (int i = 0; i < 6; ++i)
#pragma unroll
                    for (int k = 0; k < kKeys / 16; ++k)
                        umma_bf16_ts(tmem + T::kO, tmem + T::kP + kPa[i] * (kKeys / 2) + k * 8,
                                     d + (uint64_t)((kPb[i] * S::kValuePiece + k * 32) >> 4),
                                     umma_idesc_bf16(DIM), i + k > 0);
                umma_commit(o_full);
                umma_commit(&v_free[j & 1]);
            }
            if (!ok)
                fail();
            umma_commit(&drained[1]);
            if (!mbar_wait(&drained[1], 0))
                fail();
        }
      } else {
        // ================================= split =====================================
        // Half of the warps take the keys, the others the values.  A task is 32 chunks of eight
        // numbers, one 16-byte store per piece each; the next task's numbers are on their way
        // meanwhile.  Keys: chunk = eight features of a key; values: eight keys of a feature,
        // lanes along the features.
        constexpr int kTasks = kKeys * DIM / 256, kOwn = (kTasks + kSplitWarps - 1) / kSplitWarps;
        constexpr int kRow8 = DIM / 8;
        const bool values = warp >= kSplitWarp0 + kSplitWarps;
        const int w0 = (warp - kSplitWarp0) % kSplitWarps;
        // chunk i of block j
        auto load_key = [&](int j, int i, uint64_t (&x)[4]) {
            const bool in = j * kKeys + i / kRow8 < vis_max;
            const ulonglong2* src =
                reinterpret_cast<const ulonglong2*>(kc + (size_t)j * kKeys * DIM + 8 * i);
            const ulonglong2 z = make_ulonglong2(0ull, 0ull);
            const ulonglong2 a = in ? src[0] : z, b = in ? src[1] : z;
            x[0] = a.x;
            x[1] = a.y;
            x[2] = b.x;
            x[3] = b.y;
        };
        auto load_value = [&](int j, int i, uint64_t (&x)[4]) {
            const int here = vis_max - j * kKeys - i / DIM * 8;  // of the eight keys, that exist
            const float* src = vc + ((size_t)j * kKeys + i / DIM * 8) * DIM + i % DIM;
            float f[8];
            if (here >= 8) {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    f[e] = src[e * DIM];
            } else {
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    f[e] = e < here ? src[e * DIM] : 0.f;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e)
                x[e] = b2w4_pack2(f[2 * e], f[2 * e + 1]);
        };
        auto run = [&](auto load, auto place_of, int piece, uint8_t* ring, uint64_t* full,
                       uint64_t* free) {
            uint64_t next[4];
            load(0, w0 * 32 + lane, next);
            for (int j = 0; j < steps; ++j) {
                if (j >= 2 && !warp_wait(&free[j & 1], ((j >> 1) - 1) & 1)) {
                    fail();
                    break;
                }
                uint8_t* dst = ring + (j & 1) * S::kBuf;
                uint64_t left = 0ull;
#pragma unroll
                for (int u = 0; u < kOwn; ++u) {
                    const int task = w0 + kSplitWarps * u;
                    if (task >= kTasks)
                        break;
                    uint64_t x[4] = {next[0], next[1], next[2], next[3]};
                    if (task + kSplitWarps < kTasks)
                        load(j, (task + kSplitWarps) * 32 + lane, next);
                    else
                        load(j + 1, w0 * 32 + lane, next);
                    uint8_t* to = dst + place_of(task * 32 + lane);
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        uint4 o;
                        o.x = take_piece(x[0]);
                        o.y = take_piece(x[1]);
                        o.z = take_piece(x[2]);
                        o.w = take_piece(x[3]);
                        *reinterpret_cast<uint4*>(to + p * piece) = o;
                    }
                    left |= x[0] | x[1] | x[2] | x[3];
                }
                if (left)
                    *s_odd = 1;
                // make the generic-proxy writes visible to the tensor core's async proxy
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                warp_arrive(&full[j & 1]);
            }
        };
        if (values)
            run(load_value, [&](int i) { return place(i % DIM, i / DIM); }, S::kValuePiece,
                smem + S::kV, v_full, v_free);
        else
            run(load_key,
                [&](int i) {
                    const int c = i % kRow8;
                    return (c >> 3) * 3 * S::kKeyPiece + place(i / kRow8, c & 7);
                },
                S::kKeyPiece, smem + S::kK, k_full, k_free);
      }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kScoreWarp) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                     ::"r"(tmem), "r"(512)
                     : "memory");
    }
}

template <int DIM>
int launch_dim(b2w4_ctx* ctx, const float* q, const float* k_cache, const float* v_cache,
               float* out, int tokens, int heads, int kv_heads, int past, const int* past_dev,
               int capacity, float scale) {
    static b2w4_smem_optin cfg;
    auto kern = attention_tc_kernel<DIM>;
    const int tq = kRows / (heads / kv_heads);
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, TcSmem<DIM>::kTotal, cfg));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, dim3(kv_heads, (tokens + tq - 1) / tq),
                                       dim3(kTcThreads), TcSmem<DIM>::kTotal, ctx->stream, q,
                                       k_cache, v_cache, out, tokens, heads, kv_heads, past,
                                       past_dev, capacity, scale, tq, ctx->status_dev));
    ctx->launches++;
    return B2W4_OK;
}

}  // namespace

int b2w4_launch_attention_tc(b2w4_ctx* ctx, const float* q, const float* k_cache,
                             const float* v_cache, float* out, int tokens, int heads,
                             int kv_heads, int dim, int past, const int* past_dev, int capacity,
                             float scale) {
    return dim == 64 ? launch_dim<64>(ctx, q, k_cache, v_cache, out, tokens, heads, kv_heads,
                                      past, past_dev, capacity, scale)
                     : launch_dim<128>(ctx, q, k_cache, v_cache, out, tokens, heads, kv_heads,
                                       past, past_dev, capacity, scale);
}
