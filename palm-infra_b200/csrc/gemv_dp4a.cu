// W4G128 x int8 GEMV for one activation row (decode): HBM-bound weight streaming.
// (Two and more rows go to the tensor-instruction kernel in gemv_mma.cu; the row-count
// template parameter below is kept at 1.)
//
// Arithmetic = the reference's NEON W4A8 GEMV (kernels/matmul_w4.cpp:211-295) applied row
// by row, with the activation quantiser (kernels/matmul_quant.cpp:578-641) fused in:
//   per 128-k group g:  D = sum q4*q8 (int32);  y = fma(float(D), fp32(ws*as[g]), y)
// groups ascending.  The per-32 rule (kernels/matmul_w4.cpp:785-901) is the same loop
// with one D and one activation scale per 32-k block.
//
// Data movement.  A CTA owns `tpc` consecutive 8-row tiles; their nibble stream
// (tpc * K/128 * 512 bytes, contiguous in the nibble plane) and their scales are brought
// into shared memory by bulk async copies (cp.async.bulk, one per tile, completion on an
// mbarrier per tile) that one thread issues as the first thing the kernel does.  Nothing
// is staged in registers, so the whole weight of a launch is in flight within the first
// microsecond.  A CTA uses under half of an SM's shared memory, registers and threads: two
// CTAs are resident per SM, and with programmatic dependent launch the CTAs of the NEXT
// kernel in the stream become resident and start their copies while this kernel still
// computes.  Weights never depend on the previous kernel's output; only the activation
// read waits on the predecessor (griddepcontrol.wait).
//
// Math, phase 1.  An item is four consecutive groups of one tile; warp w takes items w,
// w+W, ... of the CTA in a short, not unrolled loop (the kernel is latency-sensitive and
// runs a few microseconds: its code has to stay resident in the instruction cache).  In an
// item, lane (gl = lane/8, row = lane%8) owns group gl for one weight row, reads its four
// 16-byte chunks (a quarter warp reads 128 contiguous bytes: no bank conflicts) and the
// even/odd de-interleaved int8 activations (broadcast), and gets the group's int32 sum from
// 32 dp4a with no cross-lane reduction.  A weight word w holds 8 nibbles; two logic
// instructions split it without shifts:
//   hi = w & 0xF0F0F0F0                  odd k, bytes = 16*q as int8
//   lo = (w ^ 0x08080808) & 0x0F0F0F0F   even k, bytes = q+8 as uint8
// sum(q*a) = dp4a.u8.s8(lo, a_even) - 8*sum(a_even) + dp4a.s8.s8(hi, a_odd)/16: the last
// term is an exact multiple of 16 (like the NEON kernel's sdot on left-aligned nibbles and
// its fixed-point convert) and sum(a_even) comes from the quantiser, one per group.  The
// integer sum (as a float: exact) and the scale product fp32(ws*as) go to shared memory.
// Phase 2, after one barrier: one thread per (tile, weight row, activation row) runs the
// order-sensitive chain of fused multiply-adds over the groups in ascending order.
//
// A decode step's neighbours of the matmul run inside it (b2w4_step_matmul), because as launches
// of their own they cost 2 to 3 us each, all of it latency:
//   NORM          the row (up to 4096 values) is made here, x = rms_norm(residual + update):
//                 every CTA sums the squares of the whole row (10 KB from L2) and the first one
//                 writes the new residual, to another buffer than the one that the others still
//                 read.  For a launch of one wave; where CTAs follow one another on an SM the
//                 repeated sum costs more than a launch (an lm_head of 2111 CTAs: 46 -> 65 us)
//   kModeSwiglu   a CTA takes as many tiles of the up rows as of the gate rows, the same ones,
//                 and stores silu(gate) * up
#include <cooperative_groups.h>

#include "b200w4_internal.cuh"

namespace {

// one activation row: 16 warps of <= 64 registers; more rows keep more integer sums in
// registers: 8 warps of <= 128 registers.  Either way two CTAs share an SM.
__host__ __device__ constexpr int gemv_warps(int mt) { return mt == 1 ? 16 : 8; }
constexpr int kMaxTpc = 16, kWideTpc = 24;  // tiles per CTA; of thirty-two warps
constexpr unsigned kSpinLimit = 1u << 22;  // bounded waits: give up, flag, return
constexpr unsigned long long kWaitLimitCycles = 4000000000ull;  // SM cycles: about 2 s
constexpr int kTpGatherThreads = 256;

struct GemvArgs {
    const uint4* nib;
    const void* scl;
    const float* x;
    float* y;
    int32_t* sums;  // optional [m][n][groups or 4*groups]
    int* status;    // device status word: set when a bounded wait gives up
    int lda, ldc, m, n, k, groups, tiles;
    int tpc;       // tiles per CTA
    int ipt_magic; // item / items-per-tile == (item * ipt_magic) >> 16, or 0: divide
    int d_stride;  // ints between the integer sums of consecutive tiles (padded)
    int activation, act_n_begin, act_n_len;
    b2w4_tp_args tp;  // tensor-parallel epilogue (world == 0: off)
    b2w4_top1_args top1;  // greedy-token epilogue (MODE 2)
    b2w4_norm_args norm;  // NORM: how the row is made
    bool swiglu;          // kModeSwiglu asked for
};
// Kernel modes: plain, with the int32 group sums written out, with the greedy-token epilogue,
// with SwiGLU over the two halves of the weight's rows.
constexpr int kModePlain = 0, kModeSums = 1, kModeTop1 = 2, kModeSwiglu = 3;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// global -> shared bulk copy (the TMA engine, untiled form); both addresses 16-byte
// aligned, size a multiple of 16
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// SM cycle counter: cheap to read (the global nanosecond timer is not), good enough to
// bound a wait
__device__ __forceinline__ unsigned long long wait_clock() {
    return (unsigned long long)clock64();
}
// Waits for a phase of an mbarrier; false when the iteration or the time limit runs out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity = 0) {
    if (mbar_try_wait(bar, parity))
        return true;
    const unsigned long long t0 = wait_clock();
    for (unsigned spins = 0; spins < kSpinLimit; ++spins) {
        if (mbar_try_wait(bar, parity))
            return true;
        if ((spins & 63) == 63 && wait_clock() - t0 > kWaitLimitCycles)
            return false;
    }
    return false;
}

// uint8 x int8 dot of four byte pairs
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}

// Where a group's codes lie: its four 32-blocks (16 even-k codes, then 16 odd-k codes) in an order
// that turns with the group, block s at place s ^ (g % 4).  The four groups that a warp reads with
// one load are 128 bytes apart and would share their banks (a load took four passes, and the
// shared-memory pipe was busy for 49 % of an lm_head).  us per launch, graph replay: [151936, 2560]
// 41.0 -> 39.7, [19456, 2560] 7.46 -> 7.14, [6144, 2560] 3.60 -> 3.39, [9728, 2560] 4.35 -> 4.23,
// [2560, 4096] 3.84 -> 3.74; a decode step of eight layers behind 300 keys 330.5 -> 324.2.
__device__ __forceinline__ int code_place(int s, int g) { return s ^ (g & 3); }

// Integer sum of one weight row and group: wt = the row's four 16-byte chunks (one every eight
// uint4), qa = the group's even / odd de-interleaved codes, es = -8 * sum of the even-k codes.
__device__ __forceinline__ int group_sum(const uint4* wt, const uint4* qa, int es, int g) {
    int pt = es, qt = 0;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const int at = code_place(s, g) * 2;
        const uint4 w = wt[s * 8], ae = qa[at], ao = qa[at + 1];
        int p = dp4a_us((w.x ^ 0x08080808u) & 0x0F0F0F0Fu, ae.x, 0);
        int q = __dp4a((int)(w.x & 0xF0F0F0F0u), (int)ao.x, 0);
        p = dp4a_us((w.y ^ 0x08080808u) & 0x0F0F0F0Fu, ae.y, p);
        q = __dp4a((int)(w.y & 0xF0F0F0F0u), (int)ao.y, q);
        p = dp4a_us((w.z ^ 0x08080808u) & 0x0F0F0F0Fu, ae.z, p);
        q = __dp4a((int)(w.z & 0xF0F0F0F0u), (int)ao.z, q);
        p = dp4a_us((w.w ^ 0x08080808u) & 0x0F0F0F0Fu, ae.w, p);
        q = __dp4a((int)(w.w & 0xF0F0F0F0u), (int)ao.w, q);
        pt += p;
        qt += q;
    }
    return pt + (qt >> 4);  // qt sums 16*q4*a: an exact multiple of 16
}

// the fused activations carry fp64 exp / tanh code: keep one out-of-line copy
__device__ __noinline__ float gemv_activation(float v, int act) {
    return b2w4_activation(v, act);
}

// WARPS: of a CTA; sixteen, two CTAs per SM, or the double and one.
template <int MT, bool SCL16, bool A32, int MODE, bool NORM = false, int WARPS = gemv_warps(MT)>
__global__ void __launch_bounds__(WARPS * 32, WARPS > 16 ? 1 : 2)
gemv_w4a8_kernel(const GemvArgs a) {
    constexpr int kWarps = WARPS;
    constexpr int kThreads = kWarps * 32;
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int SPG = A32 ? 4 : 1;  // integer sums per group
    const int G = a.groups, K = a.k;
    const int tile_bytes = G * 512;
    const int scl_tile_bytes = G * 8 * (SCL16 ? 2 : 4);
    // shared-memory carve-up (every region a multiple of 16 bytes)
    uint8_t* s_w = smem;                                   // [tpc][G][512]
    uint8_t* s_scl = s_w + (size_t)a.tpc * tile_bytes;     // [tpc][G][8] fp16|fp32
    uint4* s_qa = reinterpret_cast<uint4*>(s_scl + (size_t)a.tpc * scl_tile_bytes);  // [MT][K]
    float* s_as = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(s_qa) + (size_t)MT * K);
    // per (tile, group, [32-block], activation row, weight row): the integer sum as a float
    // (exact: |sum| < 2^24) and the scale product it is multiplied with
    int* s_es = reinterpret_cast<int*>(s_as + MT * G * SPG);  // -8 * sum of the even-k codes
    float* s_d = reinterpret_cast<float*>(s_es + MT * G * SPG);  // [tpc][G][SPG][MT][8] + pad
    float* s_sc = s_d + (size_t)a.tpc * a.d_stride;        // same shape
    // NORM: a copy of the row, where the sums come later
    float* s_row = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(s_d) + 15) & ~uintptr_t(15));
    const uintptr_t sums_end = reinterpret_cast<uintptr_t>(s_sc + (size_t)a.tpc * a.d_stride);
    const uintptr_t row_end = NORM ? reinterpret_cast<uintptr_t>(s_row + K) : 0;
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(
        ((row_end > sums_end ? row_end : sums_end) + 7) & ~uintptr_t(7));

    constexpr bool SUMS = MODE == kModeSums;
    __shared__ unsigned long long s_top1[8];
    if (MODE == kModeTop1 && threadIdx.x < 8)
        s_top1[threadIdx.x] = 0ull;  // barriers follow before the epilogue uses it
    unsigned long long top1_best = 0ull;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gl = lane >> 3, row = lane & 7;
    // SwiGLU: half the CTA's tiles are gate tiles, the other half the up tiles of the same rows
    constexpr bool SWIGLU = MODE == kModeSwiglu;
    const int tile0 = blockIdx.x * (SWIGLU ? a.tpc / 2 : a.tpc);
    const int run = SWIGLU ? min(a.tpc / 2, a.tiles / 2 - tile0) : min(a.tpc, a.tiles - tile0);
    const int ntile = SWIGLU ? 2 * run : run;

    // Let the next kernel in the stream become resident and start its own weight copies.
    b2w4_pdl_launch_dependents();

    // ---- weight stream: issued before anything else, independent of the predecessor ----
    if (warp == 0) {
        // lane t arms and fills tile t's barrier; lane ntile does the scales
        if (lane <= ntile)
            mbar_init(&s_bar[lane], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        if (lane < ntile) {
            const int tile = lane < run ? tile0 + lane : a.tiles / 2 + tile0 + lane - run;
            mbar_expect_tx(&s_bar[lane], (uint32_t)tile_bytes);
            bulk_g2s(s_w + (size_t)lane * tile_bytes,
                     reinterpret_cast<const uint8_t*>(a.nib) + (size_t)tile * tile_bytes,
                     (uint32_t)tile_bytes, &s_bar[lane]);
        } else if (lane == ntile) {
            const uint8_t* scl = reinterpret_cast<const uint8_t*>(a.scl);
            const uint32_t run_bytes = (uint32_t)(run * scl_tile_bytes);
            mbar_expect_tx(&s_bar[ntile], SWIGLU ? 2 * run_bytes : run_bytes);
            bulk_g2s(s_scl, scl + (size_t)tile0 * scl_tile_bytes, run_bytes, &s_bar[ntile]);
            if (SWIGLU)
                bulk_g2s(s_scl + run_bytes, scl + (size_t)(a.tiles / 2 + tile0) * scl_tile_bytes,
                         run_bytes, &s_bar[ntile]);
        }
    }

    // NORM: the norm's weights may be the work of the kernel in front, too, so they are read after
    // the wait; before it they are only brought to L2 (read before it, a decode step of eight
    // layers takes 327.6 us instead of 331.5)
    if (NORM && blockIdx.x == 0 && threadIdx.x < G * 4)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a.norm.weight + threadIdx.x * 32));
    b2w4_pdl_wait();  // activations come from the previous kernel

    // Tensor-parallel exchange number: one more than the count of completed gathers, kept in
    // the first word of this rank's staging buffer (written by the gather kernel).
    unsigned tp_exchange = 0;
    if (a.tp.world != 0)
        tp_exchange =
            *reinterpret_cast<const volatile unsigned*>(a.tp.stage_peer[a.tp.rank]) + 1u;

    // ---- fused activation quantiser: one half-warp per (activation row, group) ----------
    // lane h of the half-warp holds k = 8h .. 8h+7 of the group (a quarter of a 32-block)
    {
        const int half = lane >> 4, h = lane & 15;
        const int n_q = a.m * G;
        auto load8 = [](const float* p, float (&v)[8]) {
            const float4 lo = *reinterpret_cast<const float4*>(p);
            const float4 hi = *reinterpret_cast<const float4*>(p + 4);
            v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
            v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        };
        auto store8 = [](float* p, const float (&v)[8]) {
            *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
            *reinterpret_cast<float4*>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
        };
        // NORM: residual + update, the row's sum of squares, then (v * r) * weight: the bits of
        // b2w4_add_rms_norm, whose 256 threads each add every 256th square.  A half-warp's one
        // group stays in registers; the squares are taken from a copy in shared memory.
        float kept[8], kept_w[8], rms = 0.f;
        if (NORM) {
            __shared__ float s_ss[8];
            const int g = warp * 2 + half, at = g * 128 + h * 8;
            if (g < G) {
                load8(a.norm.residual + at, kept);
                if (a.norm.update) {
                    float u[8];
                    load8(a.norm.update + at, u);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        kept[i] = __fadd_rn(kept[i], u[i]);
                }
                store8(s_row + at, kept);
                load8(a.norm.weight + at, kept_w);  // arrives under the sum of squares
                if (blockIdx.x == 0 && a.norm.residual_out)
                    store8(a.norm.residual_out + at, kept);
            }
            __syncthreads();
            if (warp < 8) {
                float ss = 0.f;
#pragma unroll 10
                for (int d = threadIdx.x; d < K; d += 256) {
                    const float v = s_row[d];
                    ss = __fadd_rn(ss, __fmul_rn(v, v));
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
                    ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, off));
                if (lane == 0)
                    s_ss[warp] = ss;
            }
            __syncthreads();
            float ss = 0.f;
#pragma unroll
            for (int w = 0; w < 8; ++w)
                ss = __fadd_rn(ss, s_ss[w]);
            rms = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)K), a.norm.eps)));
        }
        const bool vec_x = (reinterpret_cast<uintptr_t>(a.x) & 15) == 0 && (a.lda & 3) == 0;
        // the trip count is the same for both halves of the warp (the shuffles below name
        // all 32 lanes); a half without an item works on zeros and stores nothing
#pragma unroll 1
        for (int base = warp * 2; base < n_q; base += kWarps * 2) {
            const int item = base + half;
            const bool live = item < n_q;
            const int mi = live ? item / G : 0, g = live ? item % G : 0;
            const float* src = a.x + (size_t)mi * a.lda + (size_t)g * 128 + h * 8;
            float v[8];
            if (NORM) {  // one pass: this half-warp's group
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    v[i] = live ? __fmul_rn(__fmul_rn(kept[i], rms), kept_w[i]) : 0.f;
                if (blockIdx.x == 0 && a.norm.hidden_out && live)
                    store8(a.norm.hidden_out + g * 128 + h * 8, v);
            } else if (live && vec_x) {  // two 16-byte loads instead of eight scalar ones
                load8(src, v);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    v[i] = live ? src[i] : 0.f;
            }
            float amax = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i)
                amax = fmaxf(amax, fabsf(v[i]));
            // max is exact and order-free: the butterfly gives the sequential loop's value
#pragma unroll
            for (int off = (A32 ? 2 : 8); off > 0; off >>= 1)
                amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
            float scale, inv;
            b2w4_quant_params(amax, scale, inv);
            int c[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                c[i] = b2w4_quant_code(v[i], inv);
            int esum = c[0] + c[2] + c[4] + c[6];  // integer: order-free
#pragma unroll
            for (int off = (A32 ? 2 : 8); off > 0; off >>= 1)
                esum += __shfl_xor_sync(0xffffffffu, esum, off);
            if (!live)
                continue;
            if (A32) {
                if ((h & 3) == 0) {
                    s_as[mi * G * 4 + g * 4 + (h >> 2)] = scale;
                    s_es[mi * G * 4 + g * 4 + (h >> 2)] = -8 * esum;
                }
            } else if (h == 0) {
                s_as[mi * G + g] = scale;
                s_es[mi * G + g] = -8 * esum;
            }
            // 32-block h/4 is stored as 16 even-k codes then 16 odd-k codes
            uint8_t* blk = reinterpret_cast<uint8_t*>(s_qa) + (size_t)mi * K + (size_t)g * 128 +
                           code_place(h >> 2, g) * 32;
            const int j = (h & 3) * 4;
            *reinterpret_cast<char4*>(blk + j) = make_char4(
                (signed char)c[0], (signed char)c[2], (signed char)c[4], (signed char)c[6]);
            *reinterpret_cast<char4*>(blk + 16 + j) = make_char4(
                (signed char)c[1], (signed char)c[3], (signed char)c[5], (signed char)c[7]);
        }
    }
    __syncthreads();  // quantised activations and barrier inits visible to all

    // ---- phase 1: integer group sums ---------------------------------------------------
    const int ipt = (G + 3) >> 2;
    const int n_items = ntile * ipt;
    bool timed_out = !mbar_wait_bounded(&s_bar[ntile]);  // weight scales
#pragma unroll 1
    for (int it = warp; it < n_items && !timed_out; it += kWarps) {
        const int tl = a.ipt_magic ? (it * a.ipt_magic) >> 16 : it / ipt;
        const int g = (it - tl * ipt) * 4 + gl;
        if (!mbar_wait_bounded(&s_bar[tl])) {
            timed_out = true;
            break;
        }
        if (g < G) {
            const uint4* wt =
                reinterpret_cast<const uint4*>(s_w) + (tl * tile_bytes >> 4) + g * 32 + row;
            // a weight word holds 8 nibbles; two logic instructions split it without shifts:
            // odd k as 16*q (int8), even k as q+8 (uint8)
            uint32_t wl[16], wh[16];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const uint4 w = wt[s * 8];
                wl[s * 4 + 0] = (w.x ^ 0x08080808u) & 0x0F0F0F0Fu;
                wh[s * 4 + 0] = w.x & 0xF0F0F0F0u;
                wl[s * 4 + 1] = (w.y ^ 0x08080808u) & 0x0F0F0F0Fu;
                wh[s * 4 + 1] = w.y & 0xF0F0F0F0u;
                wl[s * 4 + 2] = (w.z ^ 0x08080808u) & 0x0F0F0F0Fu;
                wh[s * 4 + 2] = w.z & 0xF0F0F0F0u;
                wl[s * 4 + 3] = (w.w ^ 0x08080808u) & 0x0F0F0F0Fu;
                wh[s * 4 + 3] = w.w & 0xF0F0F0F0u;
            }
            const int slot = tl * a.d_stride + g * SPG * MT * 8 + row;
            float* dst = s_d + slot;
            float* dsc = s_sc + slot;
            const float ws =
                SCL16 ? __half2float(reinterpret_cast<const __half*>(s_scl)[(tl * G + g) * 8 + row])
                      : reinterpret_cast<const float*>(s_scl)[(tl * G + g) * 8 + row];
#pragma unroll
            for (int mi = 0; mi < MT; ++mi) {
                if (mi < a.m) {
                    const uint4* qa = s_qa + ((mi * K + g * 128) >> 4);
                    int pt = 0, qt = 0;
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        const int place = code_place(s, gl) * 2;  // g % 4 == gl
                        const uint4 ae = qa[place], ao = qa[place + 1];
                        // two independent chains per sub-block hide dp4a latency
                        int p = dp4a_us(wl[s * 4 + 0], ae.x, 0);
                        int q = __dp4a((int)wh[s * 4 + 0], (int)ao.x, 0);
                        p = dp4a_us(wl[s * 4 + 1], ae.y, p);
                        q = __dp4a((int)wh[s * 4 + 1], (int)ao.y, q);
                        p = dp4a_us(wl[s * 4 + 2], ae.z, p);
                        q = __dp4a((int)wh[s * 4 + 2], (int)ao.z, q);
                        p = dp4a_us(wl[s * 4 + 3], ae.w, p);
                        q = __dp4a((int)wh[s * 4 + 3], (int)ao.w, q);
                        if (A32) {
                            // q sums 16*q4*a: an exact multiple of 16
                            dst[(s * MT + mi) * 8] =
                                (float)(p + s_es[mi * G * 4 + g * 4 + s] + (q >> 4));
                            dsc[(s * MT + mi) * 8] =
                                __fmul_rn(ws, s_as[mi * G * 4 + g * 4 + s]);
                        } else {
                            pt += p;
                            qt += q;
                        }
                    }
                    if (!A32) {
                        dst[mi * 8] = (float)(pt + s_es[mi * G + g] + (qt >> 4));
                        dsc[mi * 8] = __fmul_rn(ws, s_as[mi * G + g]);
                    }
                }
            }
        }
    }
    if (timed_out && lane == 0)
        b2w4_report_timeout(a.status);
    __syncthreads();

    __shared__ float s_gu[SWIGLU ? kWideTpc * 8 : 1];  // gate rows, then up rows
    // ---- phase 2: fp32 chain, one thread per (tile, activation row, weight row) ---------
#pragma unroll 1
    for (int t = threadIdx.x; t < ntile * MT * 8; t += kThreads) {
        const int rr = t & 7, mi = (t >> 3) % MT, tl = t / (8 * MT);
        if (mi >= a.m)
            continue;
        const int n = (tile0 + tl) * 8 + rr;
        const float* dsrc = s_d + (size_t)tl * a.d_stride + mi * 8 + rr;
        const float* csrc = s_sc + (size_t)tl * a.d_stride + mi * 8 + rr;
        float acc = 0.f;
        // only the fused multiply-add depends on the previous step; the loads do not
#pragma unroll 10
        for (int j = 0; j < G * SPG; ++j) {
            const float dv = dsrc[j * MT * 8];
            acc = __fmaf_rn(dv, csrc[j * MT * 8], acc);
            if (SUMS && n < a.n)
                a.sums[((size_t)mi * a.n + n) * (G * SPG) + j] = (int)dv;
        }
        if (SWIGLU) {
            s_gu[t] = acc;
        } else if (n < a.n) {
            if (b2w4_act_applies(n, a.activation, a.act_n_begin, a.act_n_len, a.n))
                acc = gemv_activation(acc, a.activation);
            if (MODE == kModeTop1) {
                // the index is the row of the unsharded weight (n_offset is 0 on one GPU)
                const unsigned long long word = b2w4_top1_word(acc, a.tp.n_offset + n);
                top1_best = word > top1_best ? word : top1_best;
                if (a.y)
                    a.y[(size_t)mi * a.ldc + n] = acc;
            } else if (a.tp.world == 0) {
                a.y[(size_t)mi * a.ldc + n] = acc;
            } else {
                // The all-gather is this store: every rank's staging buffer, this GPU's own
                // included, gets (value, exchange number) as one 8-byte word over peer
                // mappings.  The word is written whole, so the reader needs no fence: an
                // entry that carries the current exchange number carries its value.
                const unsigned long long word =
                    ((unsigned long long)tp_exchange << 32) | __float_as_uint(acc);
                const size_t at = kTpStageHeader +
                                  (size_t)(tp_exchange & 1) * kTpMaxRows * a.ldc +
                                  (size_t)mi * a.ldc + a.tp.n_offset + n;
#pragma unroll
                for (int p = 0; p < kTpMaxWorld; ++p)
                    if (p < a.tp.world)
                        a.tp.stage_peer[p][at] = word;
            }
        }
    }
    if (MODE == kModeTop1)
        b2w4_top1_finish(a.top1, top1_best, (threadIdx.x >> 3) % MT, a.m, s_top1);
    if (SWIGLU) {  // the operations of b2w4_swiglu
        __syncthreads();
        for (int t = threadIdx.x; t < run * 8; t += kThreads)
            a.y[tile0 * 8 + t] = b2w4_swiglu_value(s_gu[t], s_gu[run * 8 + t]);
    }
}

// The quantiser of gemv_w4a8_kernel for groups [0, n_g) of a row, per 128 values: a half-warp per
// group, by a CTA of sixteen warps.
__device__ __forceinline__ void quantize_groups(const float* x, int n_g, uint4* s_qa, float* s_as,
                                                int* s_es) {
    constexpr int kWarps = 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int half = lane >> 4, h = lane & 15;
    const bool vec_x = (reinterpret_cast<uintptr_t>(x) & 15) == 0;
#pragma unroll 1
    for (int base = warp * 2; base < n_g; base += kWarps * 2) {
        const int g = base + half;
        const bool live = g < n_g;
        const float* src = x + (size_t)(live ? g : 0) * 128 + h * 8;
        float v[8];
        if (live && vec_x) {
            const float4 lo = *reinterpret_cast<const float4*>(src);
            const float4 hi = *reinterpret_cast<const float4*>(src + 4);
            v[0] = lo.x; v[1] = lo.y; v[2] = lo.z; v[3] = lo.w;
            v[4] = hi.x; v[5] = hi.y; v[6] = hi.z; v[7] = hi.w;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                v[i] = live ? src[i] : 0.f;
        }
        float amax = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        float scale, inv;
        b2w4_quant_params(amax, scale, inv);
        int c[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            c[i] = b2w4_quant_code(v[i], inv);
        int esum = c[0] + c[2] + c[4] + c[6];
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
            esum += __shfl_xor_sync(0xffffffffu, esum, off);
        if (!live)
            continue;
        if (h == 0) {
            s_as[g] = scale;
            s_es[g] = -8 * esum;
        }
        uint8_t* blk =
            reinterpret_cast<uint8_t*>(s_qa) + (size_t)g * 128 + code_place(h >> 2, g) * 32;
        const int j = (h & 3) * 4;
        *reinterpret_cast<char4*>(blk + j) = make_char4(
            (signed char)c[0], (signed char)c[2], (signed char)c[4], (signed char)c[6]);
        *reinterpret_cast<char4*>(blk + 16 + j) = make_char4(
            (signed char)c[1], (signed char)c[3], (signed char)c[5], (signed char)c[7]);
    }
}

// ---- long rows: the groups split over a cluster ----------------------------------------------
// A cluster of kSplit CTAs takes `tpc` tiles; CTA r quantises and multiplies groups [r * per,
// (r + 1) * per) of all of them and stores each (integer sum, scale product) into the shared
// memory of the CTA that owns the tile (tile % kSplit), which after one cluster barrier runs the
// tiles' chains over all groups in ascending order: the kernel above, its bits, with a quarter
// of the row per CTA.  What that mends where rows are long: a CTA of the kernel above holds whole
// tiles, so a weight of few long rows leaves SMs with one or two of them (an [2560, 9728] weight:
// 160 CTAs of two tiles, 12 SMs with two such CTAs), and every CTA quantises the whole row.
constexpr int kSplit = 4;
constexpr int kSplitMaxTiles = 16;
template <bool SCL16>
__global__ void __cluster_dims__(kSplit, 1, 1) __launch_bounds__(512, 2)
gemv_w4a8_split_kernel(const GemvArgs a) {
    constexpr int kWarps = 16, kScl = SCL16 ? 16 : 32;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(128) uint8_t smem[];
    const int G = a.groups, per = (G + kSplit - 1) / kSplit;
    const int rank = blockIdx.x % kSplit, tile0 = blockIdx.x / kSplit * a.tpc;
    const int ntile = min(a.tpc, a.tiles - tile0);
    const int g0 = min(G, rank * per), n_g = min(per, G - g0);
    const int owned = (a.tpc + kSplit - 1) / kSplit;
    uint8_t* s_w = smem;                                                 // [tpc][per][512]
    uint8_t* s_scl = s_w + (size_t)a.tpc * per * 512;                    // [tpc][per][8]
    uint4* s_qa = reinterpret_cast<uint4*>(s_scl + (size_t)a.tpc * per * kScl);  // [per][128]
    float* s_as = reinterpret_cast<float*>(s_qa + per * 8);              // [per]
    int* s_es = reinterpret_cast<int*>(s_as + per);                      // [per]
    float* s_d = reinterpret_cast<float*>(s_es + per);                   // [owned][d_stride]
    float* s_sc = s_d + (size_t)owned * a.d_stride;
    __shared__ uint64_t s_bar[kSplitMaxTiles];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    b2w4_pdl_launch_dependents();
    if (warp == 0) {  // lane t: tile t's share
        if (lane < ntile)
            mbar_init(&s_bar[lane], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        if (lane < ntile && n_g > 0) {
            const size_t at = (size_t)(tile0 + lane) * G + g0;
            mbar_expect_tx(&s_bar[lane], (uint32_t)n_g * (512 + kScl));
            bulk_g2s(s_w + (size_t)lane * per * 512,
                     reinterpret_cast<const uint8_t*>(a.nib) + at * 512, (uint32_t)n_g * 512,
                     &s_bar[lane]);
            bulk_g2s(s_scl + (size_t)lane * per * kScl,
                     reinterpret_cast<const uint8_t*>(a.scl) + at * kScl, (uint32_t)n_g * kScl,
                     &s_bar[lane]);
        }
    }
    b2w4_pdl_wait();  // activations come from the previous kernel
    quantize_groups(a.x + (size_t)g0 * 128, n_g, s_qa, s_as, s_es);
    // every CTA of the cluster runs before its shared memory is written from another one
    cluster.sync();

    // integer sums: an item is four consecutive groups of one tile
    const int gl = lane >> 3, row = lane & 7, ipt = (n_g + 3) >> 2;
    bool timed_out = false;
#pragma unroll 1
    for (int it = warp; it < ntile * ipt && !timed_out; it += kWarps) {
        const int tl = it / ipt, g = (it - tl * ipt) * 4 + gl;
        if (!mbar_wait_bounded(&s_bar[tl])) {
            timed_out = true;
            break;
        }
        if (g < n_g) {
            const int at = tl * per + g;
            const int d = group_sum(reinterpret_cast<const uint4*>(s_w) + at * 32 + row,
                                    s_qa + g * 8, s_es[g], gl);
            const float ws = SCL16 ? __half2float(reinterpret_cast<const __half*>(s_scl)[at * 8 + row])
                                   : reinterpret_cast<const float*>(s_scl)[at * 8 + row];
            const int slot = (tl / kSplit) * a.d_stride + (g0 + g) * 8 + row, owner = tl % kSplit;
            cluster.map_shared_rank(s_d, owner)[slot] = (float)d;
            cluster.map_shared_rank(s_sc, owner)[slot] = __fmul_rn(ws, s_as[g]);
        }
    }
    if (timed_out && lane == 0)
        b2w4_report_timeout(a.status);
    cluster.sync();

    // the owned tiles' chains: tiles rank, rank + kSplit, ...
    for (int t = threadIdx.x; t < owned * 8; t += kWarps * 32) {
        const int rr = t & 7, to = t >> 3, tl = to * kSplit + rank;
        const int n = (tile0 + tl) * 8 + rr;
        if (tl >= ntile || n >= a.n)
            continue;
        const float* dsrc = s_d + (size_t)to * a.d_stride + rr;
        const float* csrc = s_sc + (size_t)to * a.d_stride + rr;
        float acc = 0.f;
#pragma unroll 10
        for (int j = 0; j < G; ++j)
            acc = __fmaf_rn(dsrc[j * 8], csrc[j * 8], acc);
        if (b2w4_act_applies(n, a.activation, a.act_n_begin, a.act_n_len, a.n))
            acc = gemv_activation(acc, a.activation);
        a.y[n] = acc;
    }
}

// ---- weights of many rows (an lm_head): persistent CTAs ---------------------------------------
// Two CTAs per SM take an equal run of tiles each, in chunks of `tpc` tiles through a ring of
// kStreamBufs buffers: the weights of the next chunks are on their way while one is computed, and
// the row is quantised once per CTA, where CTAs of gemv_w4a8_kernel that follow one another on an SM
// each quantise it and wait for their first weights.  Sums and chains as there: its bits.  A chunk's
// chains are a warp's per four tiles (others every time) under the next chunk's integer sums.
constexpr int kStreamBufs = 3, kStreamMaxTpc = 16;
template <bool SCL16, bool TOP1>
__global__ void __launch_bounds__(512, 2) gemv_w4a8_stream_kernel(const GemvArgs a) {
    constexpr int kWarps = 16, kScl = SCL16 ? 16 : 32;
    extern __shared__ __align__(128) uint8_t smem[];
    const int G = a.groups, tile_bytes = G * 512, scl_bytes = G * kScl;
    uint8_t* s_w = smem;                                                          // [bufs][tpc][G][512]
    uint8_t* s_scl = s_w + (size_t)kStreamBufs * a.tpc * tile_bytes;              // [bufs][tpc][G][8]
    uint4* s_qa = reinterpret_cast<uint4*>(s_scl + (size_t)kStreamBufs * a.tpc * scl_bytes);
    float* s_as = reinterpret_cast<float*>(s_qa + G * 8);                         // [G]
    int* s_es = reinterpret_cast<int*>(s_as + G);                                 // [G]
    float* s_d = reinterpret_cast<float*>(s_es + G);                              // [2][tpc][d_stride]
    float* s_sc = s_d + 2 * a.tpc * a.d_stride;                                   // the same
    __shared__ uint64_t s_bar[kStreamBufs];
    __shared__ unsigned long long s_top1[8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gl = lane >> 3, row = lane & 7;
    const int begin = (int)((long long)a.tiles * blockIdx.x / gridDim.x);
    const int end = (int)((long long)a.tiles * (blockIdx.x + 1) / gridDim.x);
    const int chunks = (end - begin + a.tpc - 1) / a.tpc;
    auto issue = [&](int c) {  // one thread
        const int tile = begin + c * a.tpc, n = min(a.tpc, end - tile), b = c % kStreamBufs;
        mbar_expect_tx(&s_bar[b], (uint32_t)(n * (tile_bytes + scl_bytes)));
        bulk_g2s(s_w + (size_t)b * a.tpc * tile_bytes,
                 reinterpret_cast<const uint8_t*>(a.nib) + (size_t)tile * tile_bytes,
                 (uint32_t)(n * tile_bytes), &s_bar[b]);
        bulk_g2s(s_scl + (size_t)b * a.tpc * scl_bytes,
                 reinterpret_cast<const uint8_t*>(a.scl) + (size_t)tile * scl_bytes,
                 (uint32_t)(n * scl_bytes), &s_bar[b]);
    };

    b2w4_pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int b = 0; b < kStreamBufs; ++b)
            mbar_init(&s_bar[b], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int c = 0; c < min(kStreamBufs, chunks); ++c)
            issue(c);
    }
    if (TOP1 && threadIdx.x < 8)
        s_top1[threadIdx.x] = 0ull;
    b2w4_pdl_wait();  // activations come from the previous kernel
    quantize_groups(a.x, G, s_qa, s_as, s_es);
    __syncthreads();

    const int ipt = (G + 3) >> 2;
    unsigned long long best = 0ull;
    int waits = chunks;  // chunks that the thread waits for: all, or those before a timeout
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
        const int tile0 = begin + c * a.tpc, ntile = min(a.tpc, end - tile0), b = c % kStreamBufs;
        const uint8_t* w = s_w + (size_t)b * a.tpc * tile_bytes;
        const uint8_t* scl = s_scl + (size_t)b * a.tpc * scl_bytes;
        float* d_out = s_d + (c & 1) * a.tpc * a.d_stride;
        float* sc_out = s_sc + (c & 1) * a.tpc * a.d_stride;
        if (c < waits && !mbar_wait_bounded(&s_bar[b], c / kStreamBufs & 1)) {
            waits = c;
            b2w4_report_timeout(a.status);
        }
#pragma unroll 1
        for (int it = warp; it < ntile * ipt; it += kWarps) {
            const int tl = a.ipt_magic ? (it * a.ipt_magic) >> 16 : it / ipt;
            const int g = (it - tl * ipt) * 4 + gl;
            if (g < G) {
                const int at = tl * G + g;
                const int d = group_sum(reinterpret_cast<const uint4*>(w) + at * 32 + row,
                                        s_qa + g * 8, s_es[g], gl);
                const float ws = SCL16 ? __half2float(reinterpret_cast<const __half*>(scl)[at * 8 + row])
                                       : reinterpret_cast<const float*>(scl)[at * 8 + row];
                const int slot = tl * a.d_stride + g * 8 + row;
                d_out[slot] = (float)d;
                sc_out[slot] = __fmul_rn(ws, s_as[g]);
            }
        }
        __syncthreads();  // sums in place, the buffer is free, and so are the sums of chunk c - 1
        if (threadIdx.x == 0 && c + kStreamBufs < chunks && c < waits)
            issue(c + kStreamBufs);
        const int mine = ((warp - c) & (kWarps - 1)) * 4 + gl;  // the lane's tile
        if (mine < ntile) {
            const float* dsrc = d_out + mine * a.d_stride + row;
            const float* csrc = sc_out + mine * a.d_stride + row;
            const int n = (tile0 + mine) * 8 + row;
            float acc = 0.f;
#pragma unroll 10
            for (int j = 0; j < G; ++j)
                acc = __fmaf_rn(dsrc[j * 8], csrc[j * 8], acc);
            if (n < a.n) {
                if (b2w4_act_applies(n, a.activation, a.act_n_begin, a.act_n_len, a.n))
                    acc = gemv_activation(acc, a.activation);
                if (TOP1) {
                    const unsigned long long word = b2w4_top1_word(acc, n);
                    best = word > best ? word : best;
                }
                if (!TOP1 || a.y)
                    a.y[n] = acc;
            }
        }
    }
    // after a timeout: not gone before the copies on their way have been waited for once more
    if (threadIdx.x == 0)
        for (int c = waits; c < min(chunks, waits + kStreamBufs); ++c)
            mbar_wait_bounded(&s_bar[c % kStreamBufs], c / kStreamBufs & 1);
    if (TOP1)
        b2w4_top1_finish(a.top1, best, 0, 1, s_top1);
}

// Second half of the tensor-parallel exchange: waits (bounded) until every entry of the
// current exchange's half of the staging buffer carries the exchange number -- written by this
// GPU's own matmul (complete: this kernel is ordered after it) and by the peers' -- and unpacks
// the values into the plain output row.  The last block then advances the exchange count.
// An entry that never arrives within `wait_limit` SM cycles becomes a quiet NaN in y (never a
// stale value of an earlier exchange) and the status word reports the time-out.
__global__ void __launch_bounds__(kTpGatherThreads)
tp_gather_kernel(unsigned long long* stage, float* y, int m, int ldc, unsigned* done,
                 int* status, unsigned long long wait_limit) {
    b2w4_pdl_chain_entry();
    unsigned* count = reinterpret_cast<unsigned*>(stage);
    const unsigned exchange = *reinterpret_cast<volatile unsigned*>(count) + 1u;
    const volatile unsigned long long* src =
        stage + kTpStageHeader + (size_t)(exchange & 1) * kTpMaxRows * ldc;
    const unsigned long long t0 = wait_clock();
    bool gave_up = false;
    // the m rows of the exchange are contiguous in the half and in y
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m * ldc;
         i += gridDim.x * blockDim.x) {
        unsigned long long word = src[i];
        while ((unsigned)(word >> 32) != exchange && !gave_up) {
            if (wait_clock() - t0 > wait_limit) {
                b2w4_report_timeout(status);
                gave_up = true;
            }
            word = src[i];
        }
        y[i] = (unsigned)(word >> 32) == exchange ? __uint_as_float((unsigned)word)
                                                  : __uint_as_float(0x7FC00000u);
    }
    __syncthreads();  // every thread of the block has read the count
    if (threadIdx.x == 0 && atomicAdd(done, 1u) == gridDim.x - 1) {
        *done = 0;  // ready for the next launch
        *count = exchange;
    }
}

// Second half of the fused greedy token on one GPU: the matmul before it in the stream left
// each row's maximum word in the cells; write the tokens and clear the cells.
__global__ void top1_token_kernel(unsigned long long* cells, int32_t* token, int m) {
    b2w4_pdl_chain_entry();
    if ((int)threadIdx.x < m) {
        const unsigned long long w = atomicExch(cells + threadIdx.x, 0ull);
        token[threadIdx.x] = (int32_t)(0xFFFFFFFFu - (unsigned)w);
    }
}

// Tensor-parallel greedy token, hand-over: this rank's maximum word of every row (left in the
// cells by the matmul, with indices of the unsharded weight) goes to every rank as two tagged
// words; the cells are cleared.  Thread (row r, rank q) stores to rank q.
__global__ void __launch_bounds__(kTop1MaxRows* kTpMaxWorld)
tp_send_token_kernel(unsigned long long* cells, const b2w4_tp_args tp, int m) {
    b2w4_pdl_chain_entry();
    __shared__ unsigned long long s_word[kTop1MaxRows];
    if ((int)threadIdx.x < m)
        s_word[threadIdx.x] = atomicExch(cells + threadIdx.x, 0ull);  // read and clear
    __syncthreads();
    const unsigned exchange =
        *reinterpret_cast<const volatile unsigned*>(tp.stage_peer[tp.rank]) + 1u;
    const unsigned long long tag = (unsigned long long)exchange << 32;
    const int r = threadIdx.x / kTpMaxWorld, q = threadIdx.x % kTpMaxWorld;
    if (r < m && q < tp.world) {
        const size_t slot = kTpStageHeader + (size_t)(exchange & 1) * kTop1StageHalf +
                            ((size_t)r * kTpMaxWorld + tp.rank) * 2;
        tp.stage_peer[q][slot] = tag | (s_word[r] >> 32);
        tp.stage_peer[q][slot + 1] = tag | (s_word[r] & 0xFFFFFFFFull);
    }
}

// ... and the pick: thread (row r, rank p) waits (bounded) for rank p's words of row r, the
// block takes the largest per row -- the one-GPU order -- and advances the count.
__global__ void __launch_bounds__(kTop1MaxRows* kTpMaxWorld)
tp_gather_token_kernel(unsigned long long* stage, int32_t* token, int m, int world, int* status,
                       unsigned long long wait_limit) {
    b2w4_pdl_chain_entry();
    __shared__ unsigned long long s_best[kTop1MaxRows];
    __shared__ int s_missing[kTop1MaxRows];  // a rank's words of this row never arrived
    unsigned* count = reinterpret_cast<unsigned*>(stage);
    const unsigned exchange = *reinterpret_cast<volatile unsigned*>(count) + 1u;
    const int r = threadIdx.x / kTpMaxWorld, p = threadIdx.x % kTpMaxWorld;
    if (threadIdx.x < kTop1MaxRows) {
        s_best[threadIdx.x] = 0ull;
        s_missing[threadIdx.x] = 0;
    }
    __syncthreads();
    if (r < m && p < world) {
        const volatile unsigned long long* src =
            stage + kTpStageHeader + (size_t)(exchange & 1) * kTop1StageHalf +
            ((size_t)r * kTpMaxWorld + p) * 2;
        const unsigned long long t0 = wait_clock();
        unsigned long long hi = src[0], lo = src[1];
        bool arrived = true;
        while ((unsigned)(hi >> 32) != exchange || (unsigned)(lo >> 32) != exchange) {
            if (wait_clock() - t0 > wait_limit) {
                b2w4_report_timeout(status);
                arrived = false;
                break;
            }
            hi = src[0], lo = src[1];
        }
        if (arrived)
            atomicMax(&s_best[r], (hi << 32) | (lo & 0xFFFFFFFFull));
        else
            s_missing[r] = 1;
    }
    __syncthreads();
    // a row that lacks a rank's maximum has no token: -1, never a guess from stale words
    if ((int)threadIdx.x < m)
        token[threadIdx.x] = s_missing[threadIdx.x]
                                 ? -1
                                 : (int32_t)(0xFFFFFFFFu - (unsigned)s_best[threadIdx.x]);
    if (threadIdx.x == 0)
        *count = exchange;
}

int gemv_d_stride(int mt, int groups, bool a32) {
    // +8 ints: consecutive tiles start 8 banks apart, so phase 2's warps read without
    // bank conflicts
    return groups * (a32 ? 4 : 1) * mt * 8 + 8;
}

size_t gemv_smem_bytes(int mt, int k, int groups, int tpc, bool scl16, bool a32,
                       bool norm = false) {
    const int spg = a32 ? 4 : 1;
    const size_t sums = 2 * sizeof(float) * (size_t)tpc * gemv_d_stride(mt, groups, a32);
    const size_t row = norm ? sizeof(float) * k + 16 : 0;  // its place is the sums'
    return (size_t)tpc * groups * 512 + (size_t)tpc * groups * 8 * (scl16 ? 2 : 4) +
           (size_t)mt * k + 2 * sizeof(float) * mt * groups * spg + (row > sums ? row : sums) + 8 +
           sizeof(uint64_t) * (tpc + 1);
}

template <int MT, bool SCL16, bool A32, int MODE, bool NORM = false, int WARPS = gemv_warps(MT)>
int launch_one(b2w4_ctx* ctx, const GemvArgs& a, size_t smem) {
    auto kern = gemv_w4a8_kernel<MT, SCL16, A32, MODE, NORM, WARPS>;
    static b2w4_smem_optin configured;  // per instantiation and device
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, configured));
    cudaLaunchConfig_t cfg = {};
    const int per_cta = MODE == kModeSwiglu ? a.tpc / 2 : a.tpc;
    const int tiles = MODE == kModeSwiglu ? a.tiles / 2 : a.tiles;
    cfg.gridDim = dim3((tiles + per_cta - 1) / per_cta);
    cfg.blockDim = dim3(WARPS * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = ctx->pdl ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    B2W4_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, a));
    ctx->launches++;
    return B2W4_OK;
}

size_t gemv_split_bytes(int per, int tpc, int d_stride, bool scl16) {
    return (size_t)tpc * per * (512 + (scl16 ? 16 : 32)) + (size_t)per * (128 + 8) +
           2 * sizeof(float) * ((tpc + kSplit - 1) / kSplit) * d_stride;
}
int launch_split(b2w4_ctx* ctx, const GemvArgs& a, bool scl16, size_t smem) {
    auto kern = scl16 ? gemv_w4a8_split_kernel<true> : gemv_w4a8_split_kernel<false>;
    static b2w4_smem_optin configured[2];  // per instantiation and device
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, configured[scl16]));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern,
                                       dim3((a.tiles + a.tpc - 1) / a.tpc * kSplit), dim3(512),
                                       smem, ctx->stream, a));
    ctx->launches++;
    return B2W4_OK;
}

size_t gemv_stream_bytes(int groups, int tpc, int d_stride, bool scl16) {
    return (size_t)kStreamBufs * tpc * groups * (512 + (scl16 ? 16 : 32)) +
           (size_t)groups * (128 + 8) + 4 * sizeof(float) * (size_t)tpc * d_stride;
}
// Tiles of a chunk: as many as fit half an SM, the count whose items fill the sixteen warps' rounds
// best; 0: none fits.
int gemv_stream_tpc(int groups, bool scl16) {
    const int ipt = (groups + 3) / 4, d_stride = gemv_d_stride(1, groups, false);
    int best = 0;
    double best_fill = 0.;
    for (int t = 1; t <= kStreamMaxTpc; ++t) {
        const int items = t * ipt;
        const double fill = (double)items / ((items + 15) / 16 * 16);
        if (gemv_stream_bytes(groups, t, d_stride, scl16) <= 112 * 1024 && fill >= best_fill) {
            best = t;
            best_fill = fill;
        }
    }
    return best;
}
// The chunk with which a launch of `ctas` CTAs of gemv_w4a8_kernel goes to the persistent kernel, or
// 0: it does not.  Lines in CTAs per SM.  Time of the persistent kernel to that one, plain / greedy
// token, in a graph over weights larger than L2:
//   three tiles and more   from 3.5.  At the line K = 256 0.82 / 0.72, 512 0.88 / 0.78, 768 0.99 / 0.97,
//                          1024 1.02 / 1.00, 1280 0.92 / 0.94, 1792 0.92 / 0.93, 2560 0.96 / 0.94; at
//                          eight 0.77 / 0.73 (512), 0.80 / 0.79 (1024), 0.87 / 0.85 (2560)
//   two tiles              from 4.5.  At 3.5, 4.5 and 8: K = 2816 1.00 / 1.04, 0.96 / 0.94, 0.96 / 0.96;
//                          3584 1.01 / 1.05, 0.98 / 0.94, 0.95 / 0.94; 4096 1.02 / 1.02, 0.96 / 0.93,
//                          0.89 / 0.89
//   one tile               from 4.5, and 40 groups: the sixteen warps take 64 groups a round, and a
//                          round of fewer leaves more of them idle than the ring gives.  K = 4352
//                          (34) 1.08 / 1.10, 1.03 / 1.08, 1.10 / 1.13; 4864 (38) 1.15 / 1.17, 1.06 /
//                          1.04, 1.06 / 1.05; 5120 1.02 / 1.11, 0.95 / 0.98, 0.96 / 0.99; 5632 1.02 /
//                          1.07, 0.91 / 0.95, 0.92 / 0.97; 7680 1.02 / 1.05, 0.93 / 0.94, 0.87 / 0.87
// fp32 scales: within 0.02 of these, by the chunk they have (K = 4096 one tile, 1.06 / 1.02 at 4.5).
int gemv_stream_chunk(int groups, bool scl16, int ctas, int sm_count) {
    const int t = gemv_stream_tpc(groups, scl16);
    return 2l * ctas < (t >= 3 ? 7l : 9l) * sm_count || (t == 1 && groups < 40) ? 0 : t;
}

template <bool SCL16, bool TOP1>
int launch_stream(b2w4_ctx* ctx, const GemvArgs& a) {
    auto kern = gemv_w4a8_stream_kernel<SCL16, TOP1>;
    static b2w4_smem_optin configured;  // per instantiation and device
    const size_t smem = gemv_stream_bytes(a.groups, a.tpc, a.d_stride, SCL16);
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, configured));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, dim3(2 * ctx->sm_count), dim3(512), smem,
                                       ctx->stream, a));
    ctx->launches++;
    return B2W4_OK;
}

template <int MT>
int launch_mt(b2w4_ctx* ctx, const GemvArgs& a, bool scl16, bool a32, bool wide, size_t smem) {
    const int mode = a.sums ? kModeSums : (a.top1.cells ? kModeTop1 : kModePlain);
    if (a.swiglu || a.norm.weight) {  // a decode step: one row, per-128 rule
        if (wide && a.norm.weight)
            return scl16 ? launch_one<MT, true, false, kModeSwiglu, true, 32>(ctx, a, smem)
                         : launch_one<MT, false, false, kModeSwiglu, true, 32>(ctx, a, smem);
        if (wide)
            return scl16 ? launch_one<MT, true, false, kModeSwiglu, false, 32>(ctx, a, smem)
                         : launch_one<MT, false, false, kModeSwiglu, false, 32>(ctx, a, smem);
        if (a.swiglu && a.norm.weight)
            return scl16 ? launch_one<MT, true, false, kModeSwiglu, true>(ctx, a, smem)
                         : launch_one<MT, false, false, kModeSwiglu, true>(ctx, a, smem);
        if (a.swiglu)
            return scl16 ? launch_one<MT, true, false, kModeSwiglu>(ctx, a, smem)
                         : launch_one<MT, false, false, kModeSwiglu>(ctx, a, smem);
        return scl16 ? launch_one<MT, true, false, kModePlain, true>(ctx, a, smem)
                     : launch_one<MT, false, false, kModePlain, true>(ctx, a, smem);
    }
#define B2W4_GEMV_MODES(S, A)                                              \
    (mode == kModeSums   ? launch_one<MT, S, A, kModeSums>(ctx, a, smem)   \
     : mode == kModeTop1 ? launch_one<MT, S, A, kModeTop1>(ctx, a, smem)   \
                         : launch_one<MT, S, A, kModePlain>(ctx, a, smem))
    if (scl16)
        return a32 ? B2W4_GEMV_MODES(true, true) : B2W4_GEMV_MODES(true, false);
    return a32 ? B2W4_GEMV_MODES(false, true) : B2W4_GEMV_MODES(false, false);
#undef B2W4_GEMV_MODES
}

}  // namespace

// Whether the kernels of up to eight rows take a row this long: one tile per CTA at least, or
// (one row with SwiGLU) a gate and an up tile.
bool b2w4_gemv_fits(const b2w4_weight* w, int m, int act_rule, bool swiglu) {
    if (m > 1)
        return b2w4_gemv_mma_fits(w, m, act_rule);
    return gemv_smem_bytes(1, w->k, w->groups, swiglu ? 2 : 1, w->scales_fp16 != 0,
                           act_rule == B2W4_ACT_G32) <= 220 * 1024;
}

// What gemv_stream_chunk says, for checks without a device.
extern "C" int b2w4_gemv_stream_plan(int groups, int scales_fp16, int ctas, int sm_count) {
    return gemv_stream_chunk(groups, scales_fp16 != 0, ctas, sm_count);
}

// Rows are processed four at a time; each pass streams the weight once.
int b2w4_launch_gemv(b2w4_ctx* ctx, const b2w4_weight* w, const float* x, int lda,
                     float* y, int ldc, int m, int act_rule, int activation,
                     int act_n_begin, int act_n_len, int32_t* sums, const b2w4_tp_args* tp,
                     const b2w4_top1_args* top1, const b2w4_norm_args* norm, bool swiglu) {
    if (tp && m > kTpMaxRows)
        return b2w4_fail(ctx, B2W4_E_INVALID, "tensor-parallel epilogue: at most %d rows",
                         kTpMaxRows);
    if (m > 1)  // several rows share one pass over the weight on the tensor instruction
        return b2w4_launch_gemv_mma(ctx, w, x, lda, y, ldc, m, act_rule, activation, act_n_begin,
                                    act_n_len, sums, tp, top1);
    const bool a32 = act_rule == B2W4_ACT_G32;
    const int spg = a32 ? 4 : 1;
    const bool scl16 = w->scales_fp16 != 0;
    for (int m0 = 0; m0 < m; m0 += 4) {
        const int mc = min(4, m - m0);
        const int mt = mc == 1 ? 1 : (mc == 2 ? 2 : 4);
        GemvArgs a;
        a.nib = w->nib;
        a.scl = w->scl;
        a.x = x + (size_t)m0 * lda;
        a.y = y ? y + (size_t)m0 * ldc : nullptr;
        a.sums = sums ? sums + (size_t)m0 * w->n * w->groups * spg : nullptr;
        a.status = ctx->status_dev;
        a.lda = lda;
        a.ldc = ldc;
        a.m = mc;
        a.n = w->n;
        a.k = w->k;
        a.groups = w->groups;
        a.tiles = w->tiles;
        a.activation = activation;
        a.act_n_begin = act_n_begin;
        a.act_n_len = act_n_len;
        a.tp = b2w4_tp_args();
        if (tp)
            a.tp = *tp;
        else
            a.tp.world = 0;
        a.top1 = b2w4_top1_args();
        if (top1)
            a.top1 = *top1;
        a.norm = b2w4_norm_args();
        if (norm)
            a.norm = *norm;
        a.swiglu = swiglu;
        bool wide = false;
        // Tiles per CTA: a CTA's shared memory stays under half an SM's so that two CTAs share
        // an SM, and the launch is one wave of at most 1.75 CTAs per SM.  Measured on the
        // decode shapes of a 4B dense model (148 SMs): N=9728 K=2560 (1216 tiles) 244 CTAs
        // 4.26 us (152 CTAs 6.0, 304 CTAs needing a second wave 6.6); N=6144 (768 tiles) 256
        // CTAs 3.55 us against 192 CTAs 4.08; N=19456 (2432 tiles) 271 CTAs 7.0 us against 304
        // CTAs 8.65.
        const int per_tile = w->groups * (512 + (scl16 ? 16 : 32)) +
                             8 * gemv_d_stride(mt, w->groups, a32);
        const int budget = 113 * 1024 - mt * w->k - 8 * mt * w->groups * spg - 1024;
        int most = max(1, min(budget / per_tile, kMaxTpc));
        while (norm && most > 1 &&
               gemv_smem_bytes(mt, w->k, w->groups, most, scl16, a32, true) > 112 * 1024)
            --most;  // few tiles: the row needs more room than their sums
        int tpc = most;
        const int wave_ctas = ctx->sm_count * 7 / 4;
        const int one_wave = (w->tiles + wave_ctas - 1) / wave_ctas;
        tpc = min(tpc, max(1, one_wave));
        if (ctx->gemv_tpc_override > 0)
            tpc = min(tpc, ctx->gemv_tpc_override);
        if (swiglu) {  // gate and up tiles in pairs
            const int pairs = w->tiles / 2, ctas = (w->tiles + tpc - 1) / tpc;
            tpc = min(max(2, most / 2 * 2), 2 * ((pairs + ctas - 1) / ctas));
            // Pairs that two CTAs per SM leave to a second wave: one CTA of twice the warps per SM
            // ([19456, 2560] with the norm 10.2 -> 8.9 us; 18944 rows, the last of one wave, 8.6).
            const int all = 2 * ((pairs + ctx->sm_count - 1) / ctx->sm_count);
            wide = a.top1.cells == nullptr && !a32 && ctx->gemv_tpc_override == 0 &&
                   (pairs + tpc / 2 - 1) / (tpc / 2) > 2 * ctx->sm_count && all <= kWideTpc &&
                   gemv_smem_bytes(mt, w->k, w->groups, all, scl16, a32, norm != nullptr) <=
                       220 * 1024;
            if (wide)
                tpc = all;
        }
        auto take = [&](int tiles) {
            a.tpc = tiles;
            const int ipt = (w->groups + 3) / 4;
            a.ipt_magic = 65536 / ipt + 1;
            for (int it = 0; it < tiles * ipt; ++it)  // exact for every item of a CTA?
                if (((it * a.ipt_magic) >> 16) != it / ipt)
                    a.ipt_magic = 0;
        };
        take(tpc);
        a.d_stride = gemv_d_stride(mt, w->groups, a32);
        // Long rows, split over clusters, from 48 groups on and where the kernel above has at most
        // four tiles per CTA and all clusters run at once.  us in a graph, that kernel / split, by
        // weight rows: K = 9728 1000 5.9 / 4.2, 2560 7.8 / 6.0, 4096 8.5 / 7.6; K = 6144 4.3 / 3.7,
        // 5.6 / 4.7, 5.8 / 5.8, 6144 rows 7.2 / 7.2, 8704 9.9 / 8.3, and with a second wave 9728 10.5 /
        // 13.7, 12288 12.2 / 14.2, 20000 17.9 / 22.7; K = 5120 4.1 / 3.4, 5.0 / 4.2, 5.1 / 5.2, 6144
        // rows 6.2 / 6.4; K = 4096 3.2 / 3.2, 3.9 / 3.8, 4.1 / 4.6, 4.9 / 5.6; K = 2560 2.9 / 3.1, 3.3 /
        // 3.5, 3.3 / 3.9, 9728 rows 4.7 / 9.4.  (40 groups on up to 2560 rows would gain too; 49 to 56
        // on 4096 to 6144 lose: 6656 5.7 / 5.9, 6.5 / 6.9, 7.0 / 7.6.)
        if (!a32 && !sums && !tp && !top1 && !norm && !swiglu && ctx->gemv_tpc_override == 0 &&
            w->groups >= 48 && tpc <= 4 && b2w4_gemv_fits(w, 1, act_rule)) {
            const int per = (w->groups + kSplit - 1) / kSplit;
            // clusters in one wave of at most 1.75 CTAs per SM, two CTAs' memory per SM
            const int clusters = wave_ctas / kSplit;
            a.tpc = min(kSplitMaxTiles, (w->tiles + clusters - 1) / clusters);
            const size_t bytes = gemv_split_bytes(per, a.tpc, a.d_stride, scl16);
            if (bytes <= 113 * 1024 &&
                (w->tiles + a.tpc - 1) / a.tpc * kSplit <= 2 * ctx->sm_count)
                return launch_split(ctx, a, scl16, bytes);
            a.tpc = tpc;
        }
        // Many rows: persistent CTAs.
        if (!a32 && !sums && !tp && !norm && !swiglu && ctx->gemv_tpc_override == 0) {
            const int chunk = gemv_stream_chunk(w->groups, scl16, (w->tiles + tpc - 1) / tpc,
                                                ctx->sm_count);
            if (chunk > 0) {
                take(chunk);
                return top1 ? (scl16 ? launch_stream<true, true>(ctx, a)
                                     : launch_stream<false, true>(ctx, a))
                            : (scl16 ? launch_stream<true, false>(ctx, a)
                                     : launch_stream<false, false>(ctx, a));
            }
        }
        const size_t smem =
            gemv_smem_bytes(mt, w->k, w->groups, tpc, scl16, a32, norm != nullptr);
        if (smem > 220 * 1024)
            return b2w4_fail(ctx, B2W4_E_INVALID, "gemv: K=%d needs %zu B shared memory",
                             w->k, smem);
        int rc = launch_mt<1>(ctx, a, scl16, a32, wide, smem);  // mt == 1: see the top
        if (rc != B2W4_OK)
            return rc;
    }
    return B2W4_OK;
}

int b2w4_launch_top1_token(b2w4_ctx* ctx, unsigned long long* cells, int32_t* token, int m) {
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, top1_token_kernel, dim3(1), dim3(32), 0,
                                       ctx->stream, cells, token, m));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_launch_tp_send_token(b2w4_ctx* ctx, unsigned long long* cells, const b2w4_tp_args& tp,
                              int m) {
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, tp_send_token_kernel, dim3(1),
                                       dim3(kTop1MaxRows * kTpMaxWorld), 0, ctx->stream, cells,
                                       tp, m));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_launch_tp_gather_token(b2w4_ctx* ctx, unsigned long long* stage_local, int32_t* token,
                                int m, int world) {
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, tp_gather_token_kernel, dim3(1),
                                       dim3(kTop1MaxRows * kTpMaxWorld), 0, ctx->stream,
                                       stage_local, token, m, world, ctx->status_dev,
                                       ctx->peer_wait_cycles));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_launch_tp_gather(b2w4_ctx* ctx, unsigned long long* stage_local, float* y, int m,
                          int ldc) {
    const int blocks = max(1, min((m * ldc + kTpGatherThreads - 1) / kTpGatherThreads,
                                  ctx->sm_count));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, tp_gather_kernel, dim3(blocks),
                                       dim3(kTpGatherThreads), 0, ctx->stream, stage_local, y,
                                       m, ldc, reinterpret_cast<unsigned*>(ctx->flag_dev + 6),
                                       ctx->status_dev, ctx->peer_wait_cycles));
    ctx->launches++;
    return B2W4_OK;
}
