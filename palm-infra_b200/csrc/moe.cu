// Routed mixture-of-experts op on the GPU, Qwen3-MoE configuration (softmax top-k routing,
// no shared expert).  Stands in for kernel_qwen3_moe (reference kernels/moe.cpp:576-1129)
// and select_moe_routes (kernels/moe_routing.cpp:25-169):
//   1 router logits          hidden[T,H] x router[E,H]^T, fp16 router, fp64 accumulation
//   2 route selection        top-k by raw logit, ties to the lower expert id, softmax over
//                            the k selected logits
//   3 compaction             counting sort of the T*k routes by expert, tokens ascending
//   4 activation quantiser   int8 per 128 values, once per token (shared by its routes)
//   5 grouped gate_up GEMV   per expert, over its ragged route list  -> [routes][2I]
//   6 SwiGLU + quantiser     silu(gate) * up, int8 per 128 values    -> [routes][I]
//   7 grouped down GEMV                                              -> [routes][H]
//   8 combine                out[t] = sum_e w * y, experts in ascending id, sequential fma
// Expert matmuls use the same W4A8 arithmetic as the dense path (per-128 rule, int32 group
// sums, fp32 chain in group order), so a route's result equals a one-row GEMV of that
// expert's weight slice.  Nothing is atomically accumulated: every output is written by one
// thread in a fixed order.
#include <type_traits>

#include <cooperative_groups.h>

#include "b200w4_internal.cuh"

namespace {

constexpr unsigned kSpinLimit = 1u << 22;
constexpr unsigned long long kWaitLimitCycles = 4000000000ull;  // SM cycles: about 2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// SM cycle counter: cheap to read (the global nanosecond timer is not), good enough to
// bound a wait
__device__ __forceinline__ unsigned long long wait_clock() {
    return (unsigned long long)clock64();
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
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar) {
    if (mbar_try_wait(bar, 0))
        return true;
    const unsigned long long t0 = wait_clock();
    for (unsigned spins = 0; spins < kSpinLimit; ++spins) {
        if (mbar_try_wait(bar, 0))
            return true;
        if ((spins & 63) == 63 && wait_clock() - t0 > kWaitLimitCycles)
            return false;
    }
    return false;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes,
                                         uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// ---- 1. router logits: one warp per (4 tokens, EPW experts) -----------------------------
// fp32 activation times fp16 weight is exact in fp64 and a few thousand such terms of
// similar magnitude add without rounding, so the fp64 sum does not depend on its order;
// one rounding to fp32 at the end (the oracle accumulates the same way).  A lane takes 8
// consecutive columns per step (one 16-byte load of router halves, two of each token's
// activations); the warp's router rows are reused for its 4 tokens.
constexpr int kRouterTok = 4;
// logits of tokens t0..t0+NT-1 against experts e0..e0+EPW-1, computed by one warp.  The K loop
// is unrolled so that several steps' loads are in flight at once: with one token and one
// expert per warp (decode) the warp is a pure latency chain otherwise.
template <int EPW, int NT>
__device__ __forceinline__ void router_logits_warp(const float* __restrict__ hidden, int ldx,
                                                   int tokens, int hidden_size,
                                                   const __half* __restrict__ router,
                                                   int num_experts, float* __restrict__ logits,
                                                   int t0, int e0, int lane) {
    double acc[NT][EPW];
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < EPW; ++j)
            acc[i][j] = 0.0;
#pragma unroll (NT == 1 ? 8 : 2)
    for (int d = lane * 8; d < hidden_size; d += 256) {
        float xv[NT][8];
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            // rows past the last token repeat it: loaded, never stored
            const float* x = hidden + (size_t)min(t0 + i, tokens - 1) * ldx + d;
            const float4 lo = *reinterpret_cast<const float4*>(x);
            const float4 hi = *reinterpret_cast<const float4*>(x + 4);
            xv[i][0] = lo.x, xv[i][1] = lo.y, xv[i][2] = lo.z, xv[i][3] = lo.w;
            xv[i][4] = hi.x, xv[i][5] = hi.y, xv[i][6] = hi.z, xv[i][7] = hi.w;
        }
#pragma unroll
        for (int j = 0; j < EPW; ++j) {
            const int e = min(e0 + j, num_experts - 1);
            const uint4 raw = *reinterpret_cast<const uint4*>(router + (size_t)e * hidden_size + d);
            const __half2* h2 = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 r = __half22float2(h2[c]);
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    acc[i][j] += (double)xv[i][2 * c] * (double)r.x;
                    acc[i][j] += (double)xv[i][2 * c + 1] * (double)r.y;
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int j = 0; j < EPW; ++j) {
            double v = acc[i][j];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                v += __shfl_xor_sync(0xffffffffu, v, off);
            if (lane == 0 && t0 + i < tokens && e0 + j < num_experts)
                logits[(size_t)(t0 + i) * num_experts + e0 + j] = (float)v;
        }
}

template <int EPW>
__global__ void moe_router_logits_kernel(const float* __restrict__ hidden, int ldx, int tokens,
                                         int hidden_size, const __half* __restrict__ router,
                                         int num_experts, float* __restrict__ logits) {
    b2w4_pdl_chain_entry();
    const int eblocks = (num_experts + EPW - 1) / EPW;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    const int tblocks = (tokens + kRouterTok - 1) / kRouterTok;
    if (wid >= (long long)tblocks * eblocks)
        return;
    const int t0 = (int)(wid / eblocks) * kRouterTok, e0 = (int)(wid % eblocks) * EPW;
    router_logits_warp<EPW, kRouterTok>(hidden, ldx, tokens, hidden_size, router, num_experts,
                                        logits, t0, e0, lane);
}

// Fallback for activations whose rows are not 16-byte aligned: one warp per (token, expert),
// scalar loads.
__global__ void moe_router_logits_scalar_kernel(const float* __restrict__ hidden, int ldx,
                                                int tokens, int hidden_size,
                                                const __half* __restrict__ router,
                                                int num_experts, float* __restrict__ logits) {
    b2w4_pdl_chain_entry();
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)tokens * num_experts)
        return;
    const int t = (int)(wid / num_experts), e = (int)(wid % num_experts);
    const float* x = hidden + (size_t)t * ldx;
    const __half* r = router + (size_t)e * hidden_size;
    double acc = 0.0;
    for (int d = lane; d < hidden_size; d += 32)
        acc += (double)x[d] * (double)__half2float(r[d]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0)
        logits[(size_t)t * num_experts + e] = (float)acc;
}

// ---- 2. route selection: one warp per token ---------------------------------------------
// The reference selects by insertion with strict '>' (kernels/moe_routing.cpp:129-142): the
// result is the k largest logits in descending order, equal logits in ascending expert id,
// and a logit that is -inf or NaN never displaces the initial (expert 0, -inf) slot.  Here
// that is k rounds of a warp-wide arg-max over (logit descending, expert id ascending) with
// taken experts masked out; a round is two warp reductions (redux.sync) on integer keys.  Then the softmax over the selected logits: exp(l - l_max),
// sequential fp32 sum, times 1/sum (:157-166).
constexpr int kMaxTopK = 16;
constexpr int kSelectMaxExperts = 1024;  // 32 lanes x 32 logits in registers

// The first `rounds` routes of a token, by one warp: lane j gets the j-th expert and its logit
// (lanes from `rounds` on: expert 0, -inf).  NS = logits per lane (32 * NS >= experts).
template <int NS>
__device__ __forceinline__ int pick_routes_warp(const float* row, int num_experts, int rounds,
                                                int lane, float& logit) {
    // the lane's logits (experts lane, lane+32, ...) stay in registers for all k rounds
    float mine[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s)
        mine[s] = lane + 32 * s < num_experts ? row[lane + 32 * s] : NAN;
    float my_v = -INFINITY;   // lane j keeps the j-th selected logit
    int my_e = 0;
    // Order-preserving integer key of a logit: larger float <=> larger key, -0 counted as +0
    // like the float comparison does; NaN and -inf get key 0, which never qualifies (the
    // insertion's strict '>' against its initial -inf).
    uint32_t key[NS];
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const float v = __fadd_rn(mine[s], 0.f);
        const uint32_t u = __float_as_uint(v);
        key[s] = !(v > -INFINITY) ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
    }
    for (int j = 0; j < rounds; ++j) {
        uint32_t bk = 0u;
        int bs = 0;
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if (key[s] > bk) {  // strict: of equal logits the lower expert id stays
                bk = key[s];
                bs = s;
            }
        // two warp reductions: the largest key, then the lowest expert id that holds it
        const uint32_t wk = __reduce_max_sync(0xffffffffu, bk);
        const uint32_t we = __reduce_min_sync(
            0xffffffffu, (wk != 0u && bk == wk) ? (uint32_t)(lane + 32 * bs) : 0xffffffffu);
        if (wk != 0u && (int)(we & 31u) == lane) {
#pragma unroll
            for (int s = 0; s < NS; ++s)
                if (s == (int)(we >> 5))
                    key[s] = 0u;  // taken
        }
        if (lane == j && wk != 0u) {  // the key gives the logit back, bit for bit
            my_v = __uint_as_float((wk & 0x80000000u) ? (wk ^ 0x80000000u) : ~wk);
            my_e = (int)we;
        }
    }
    logit = my_v;
    return my_e;
}

// dispatch on the number of experts
__device__ __forceinline__ int pick_routes_any(const float* row, int num_experts, int rounds,
                                               int lane, float& logit) {
    if (num_experts <= 128)
        return pick_routes_warp<4>(row, num_experts, rounds, lane, logit);
    if (num_experts <= 256)
        return pick_routes_warp<8>(row, num_experts, rounds, lane, logit);
    if (num_experts <= 512)
        return pick_routes_warp<16>(row, num_experts, rounds, lane, logit);
    return pick_routes_warp<kSelectMaxExperts / 32>(row, num_experts, rounds, lane, logit);
}

// Routes of token t, by one warp; also returns lane j's expert (lanes >= top_k: undefined).
template <int NS>
__device__ __forceinline__ int select_routes_warp(const float* logits, int t,
                                                  int num_experts, int top_k,
                                                  int32_t* __restrict__ idx,
                                                  float* __restrict__ weights, int lane) {
    float my_v;
    const int my_e = pick_routes_warp<NS>(logits + (size_t)t * num_experts, num_experts, top_k,
                                          lane, my_v);
    const float maximum = __shfl_sync(0xffffffffu, my_v, 0);
    // exp in fp64 and one rounding: agrees with a correctly rounded expf
    const float ex = lane < top_k ? (float)exp((double)__fsub_rn(my_v, maximum)) : 0.f;
    float sum = 0.f;
    for (int j = 0; j < top_k; ++j)
        sum = __fadd_rn(sum, __shfl_sync(0xffffffffu, ex, j));
    const float inverse = sum > 0.f ? __fdiv_rn(1.f, sum) : 0.f;
    if (lane < top_k) {
        idx[(size_t)t * top_k + lane] = my_e;
        weights[(size_t)t * top_k + lane] = __fmul_rn(ex, inverse);
    }
    return my_e;
}

// dispatch on the number of experts
__device__ __forceinline__ int select_routes_any(const float* logits, int t, int num_experts,
                                                 int top_k, int32_t* __restrict__ idx,
                                                 float* __restrict__ weights, int lane) {
    if (num_experts <= 128)
        return select_routes_warp<4>(logits, t, num_experts, top_k, idx, weights, lane);
    if (num_experts <= 256)
        return select_routes_warp<8>(logits, t, num_experts, top_k, idx, weights, lane);
    if (num_experts <= 512)
        return select_routes_warp<16>(logits, t, num_experts, top_k, idx, weights, lane);
    return select_routes_warp<kSelectMaxExperts / 32>(logits, t, num_experts, top_k, idx, weights,
                                                      lane);
}

__global__ void moe_select_routes_kernel(const float* __restrict__ logits, int tokens,
                                         int num_experts, int top_k, int32_t* __restrict__ idx,
                                         float* __restrict__ weights) {
    b2w4_pdl_chain_entry();
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t >= tokens)
        return;
    select_routes_any(logits, t, num_experts, top_k, idx, weights, lane);
}

// ---- 3. compaction: a block per expert -----------------------------------------------------
// counts, exclusive offsets, and per expert its routes in ascending token order
// (kernels/moe.cpp:759-776).  pos[t][j] = the compact position of token t's j-th route;
// slots[y] = (expert, first route, one past its last route) of the y-th expert that has routes,
// ascending; empty (0, 0, 0) from the number of such experts on: what a grouped-matmul CTA
// needs to start, in one 16-byte load.
// A block reads all routes: its expert's first position is the number of routes of lower experts,
// its slot the number of lower experts that have any, so no block waits for another.  Thread t
// owns a run of consecutive routes, a scan over the threads places its routes.  (In one block,
// with the counts of all experts, the same took 12 us for 2048 routes over 128 experts.)
constexpr int kCompactThreads = 256;
__global__ void __launch_bounds__(kCompactThreads)
moe_compact_kernel(const int32_t* __restrict__ idx, int tokens, int top_k, int num_experts,
                   int32_t* __restrict__ offsets, int32_t* __restrict__ route_token,
                   int32_t* __restrict__ pos, int4* __restrict__ slots) {
    b2w4_pdl_chain_entry();
    __shared__ unsigned s_has[kSelectMaxExperts / 32];  // experts with routes
    __shared__ int s_warp[kCompactThreads / 32][2];
    const int e = blockIdx.x, routes = tokens * top_k;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int w = threadIdx.x; w < (num_experts + 31) / 32; w += kCompactThreads)
        s_has[w] = 0;
    __syncthreads();
    const int per = (routes + kCompactThreads - 1) / kCompactThreads;
    const int i0 = min(routes, (int)threadIdx.x * per), i1 = min(routes, i0 + per);
    int lower = 0, mine = 0;
    for (int i = i0; i < i1; ++i) {
        const int x = idx[i];
        if (x >= 0) {
            lower += x < e;
            mine += x == e;
            if (!(s_has[x >> 5] >> (x & 31) & 1))  // most are there already
                atomicOr(&s_has[x >> 5], 1u << (x & 31));
        }
    }
    int first = mine;  // inclusive scan of `mine`, sum of `lower`
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int f = __shfl_up_sync(0xffffffffu, first, off);
        if (lane >= off)
            first += f;
        lower += __shfl_xor_sync(0xffffffffu, lower, off);
    }
    if (lane == 31) {
        s_warp[warp][0] = first;
        s_warp[warp][1] = lower;
    }
    __syncthreads();
    int before = 0, count = 0, start = 0;
#pragma unroll
    for (int w = 0; w < kCompactThreads / 32; ++w) {
        before += w < warp ? s_warp[w][0] : 0;
        count += s_warp[w][0];
        start += s_warp[w][1];
    }
    int at = start + before + first - mine;
    for (int i = i0; i < i1 && mine > 0; ++i)
        if (idx[i] == e) {
            route_token[at] = i / top_k;
            pos[i] = at++;
        }
    if (threadIdx.x == 0) {
        int rank = 0, active = 0;  // experts with routes below this one, and in all
        for (int w = 0; w < (num_experts + 31) / 32; ++w) {
            const int n = __popc(s_has[w]);
            active += n;
            rank += w < (e >> 5) ? n : w == (e >> 5) ? __popc(s_has[w] & ((1u << (e & 31)) - 1)) : 0;
        }
        offsets[e] = start;
        if (e == num_experts - 1)
            offsets[num_experts] = start + count;
        if (count > 0)
            slots[rank] = make_int4(e, start, start + count, 0);
        else
            slots[active + e - rank] = make_int4(0, 0, 0, 0);
    }
}

// ---- 1-4 fused for a few tokens (decode) ---------------------------------------------------
// One launch instead of four: every warp of the grid quantises its share of the hidden rows
// and computes its share of the router logits; the block that arrives last at a counter (no
// block waits for another) selects the routes, one warp per token, and compacts them.  Same
// device functions, same bits as the separate kernels.  !SELECT: it ends with the logits, see
// GroupedSmallArgs.
constexpr int kFusedSwigluTokens = 4;
constexpr int kFusedTokens = 8;
constexpr int kFusedRoutes = 128;
constexpr int kFusedThreads = 128;
template <bool SELECT>
__global__ void __launch_bounds__(kFusedThreads)
moe_route_fused_kernel(const float* __restrict__ hidden, int ldx, int tokens, int hidden_size,
                       const __half* __restrict__ router, int num_experts, int top_k,
                       float* logits, int32_t* __restrict__ idx, float* __restrict__ weights,
                       int32_t* __restrict__ offsets, int32_t* __restrict__ route_token,
                       int32_t* __restrict__ pos, int4* __restrict__ slots,
                       int8_t* __restrict__ q_hidden, float* __restrict__ as_hidden,
                       int* __restrict__ arrivals) {
    b2w4_pdl_chain_entry();
    __shared__ int s_last;
    __shared__ int s_route[kFusedRoutes];  // expert of route i = (token, j)
    extern __shared__ int s_cnt[];         // [E+1]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gwarp = blockIdx.x * (kFusedThreads / 32) + warp;
    const int nwarps = gridDim.x * (kFusedThreads / 32);
    // hidden rows -> int8, one warp per (token, 128-group), codes in tensor-operand order
    const int G = hidden_size >> 7;
    for (int task = gwarp; task < tokens * G; task += nwarps) {
        const int row = task / G, g = task - row * G;
        const float4 v = *reinterpret_cast<const float4*>(hidden + (size_t)row * ldx +
                                                          (size_t)g * 128 + lane * 4);
        float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
        float scale, inv;
        b2w4_quant_params(amax, scale, inv);
        const int c0 = b2w4_quant_code(v.x, inv), c1 = b2w4_quant_code(v.y, inv);
        const int c2 = b2w4_quant_code(v.z, inv), c3 = b2w4_quant_code(v.w, inv);
        if (lane == 0)
            as_hidden[(size_t)row * G + g] = scale;
        int8_t* blk = q_hidden + (size_t)row * hidden_size + (size_t)g * 128 +
                      ((lane & 7) >> 1) * 32 + (lane >> 3) * 4 + (lane & 1) * 2;
        *reinterpret_cast<char2*>(blk) = make_char2((signed char)c0, (signed char)c2);
        *reinterpret_cast<char2*>(blk + 16) = make_char2((signed char)c1, (signed char)c3);
    }
    // router logits, one warp per expert and block of four tokens
    for (int e = gwarp; e < num_experts; e += nwarps) {
        if (tokens == 1)
            router_logits_warp<1, 1>(hidden, ldx, tokens, hidden_size, router, num_experts, logits,
                                     0, e, lane);
        else
            for (int t0 = 0; t0 < tokens; t0 += kRouterTok)
                router_logits_warp<1, kRouterTok>(hidden, ldx, tokens, hidden_size, router,
                                                  num_experts, logits, t0, e, lane);
    }
    if constexpr (!SELECT)
        return;
    // arrival: the last block to get here sees every block's logits
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(arrivals, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    for (int t = warp; t < tokens; t += kFusedThreads / 32) {
        const int e = select_routes_any(logits, t, num_experts, top_k, idx, weights, lane);
        if (lane < top_k)
            s_route[t * top_k + lane] = e;
    }
    for (int e = threadIdx.x; e <= num_experts; e += kFusedThreads)
        s_cnt[e] = 0;
    for (int y = threadIdx.x; y < num_experts; y += kFusedThreads)
        slots[y] = make_int4(0, 0, 0, 0);  // experts with routes overwrite theirs below
    __syncthreads();
    const int routes = tokens * top_k;
    if (threadIdx.x < routes)
        atomicAdd(&s_cnt[s_route[threadIdx.x]], 1);  // integer counts: order-free
    __syncthreads();
    // exclusive scan of the counts (and of "has routes") over the experts, a block-wide chunk
    // of experts at a time; then thread e places its routes in token order
    __shared__ int s_wsum[kFusedThreads / 32][2];
    int carry_run = 0, carry_rank = 0;
    for (int base = 0; base <= num_experts; base += kFusedThreads) {
        const int e = base + threadIdx.x;
        const int c = e < num_experts ? s_cnt[e] : 0;
        int run = c, rank = c > 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {  // inclusive scan inside the warp
            const int r = __shfl_up_sync(0xffffffffu, run, off);
            const int k = __shfl_up_sync(0xffffffffu, rank, off);
            if (lane >= off) {
                run += r;
                rank += k;
            }
        }
        if (lane == 31) {
            s_wsum[warp][0] = run;
            s_wsum[warp][1] = rank;
        }
        __syncthreads();
        int wrun = carry_run, wrank = carry_rank, trun = 0, trank = 0;
#pragma unroll
        for (int w = 0; w < kFusedThreads / 32; ++w) {
            if (w < warp) {
                wrun += s_wsum[w][0];
                wrank += s_wsum[w][1];
            }
            trun += s_wsum[w][0];
            trank += s_wsum[w][1];
        }
        run += wrun - c;          // exclusive
        rank += wrank - (c > 0);
        if (e <= num_experts) {
            offsets[e] = run;
            if (e < num_experts && c > 0) {
                slots[rank] = make_int4(e, run, run + c, 0);
                for (int i = 0; i < routes; ++i)
                    if (s_route[i] == e) {
                        route_token[run] = i / top_k;
                        pos[i] = run;
                        ++run;
                    }
            }
        }
        carry_run += trun;
        carry_rank += trank;
        __syncthreads();
    }
    if (threadIdx.x == 0)
        *arrivals = 0;  // ready for the next launch
}

// Hidden rows for the grouped matmul, one warp per (token, 128-group): codes in tensor-operand
// order and scales per 128 values, and (q32 != null) per 32 values as well.
__global__ void moe_quantize_hidden_kernel(const float* __restrict__ hidden, int ldx, int tokens,
                                           int hidden_size, int8_t* __restrict__ q,
                                           float* __restrict__ scales,
                                           int8_t* __restrict__ q32,
                                           float* __restrict__ scales32) {
    b2w4_pdl_chain_entry();
    const int G = hidden_size >> 7;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)tokens * G)
        return;
    const int row = (int)(wid / G), g = (int)(wid % G);
    const float* src = hidden + (size_t)row * ldx + (size_t)g * 128 + lane * 4;
    const float v[4] = {src[0], src[1], src[2], src[3]};
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)  // the lane's 32-block: eight lanes
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    const size_t at = (size_t)row * hidden_size + (size_t)g * 128 + ((lane & 7) >> 1) * 32 +
                      (lane >> 3) * 4 + (lane & 1) * 2;
    auto store = [&](float max, bool a32, int8_t* dst, float* scale_dst) {
        float scale, inv;
        b2w4_quant_params(max, scale, inv);
        const int c0 = b2w4_quant_code(v[0], inv), c1 = b2w4_quant_code(v[1], inv);
        const int c2 = b2w4_quant_code(v[2], inv), c3 = b2w4_quant_code(v[3], inv);
        if (a32 ? (lane & 7) == 0 : lane == 0)
            scale_dst[a32 ? lane >> 3 : 0] = scale;
        *reinterpret_cast<char2*>(dst) = make_char2((signed char)c0, (signed char)c2);
        *reinterpret_cast<char2*>(dst + 16) = make_char2((signed char)c1, (signed char)c3);
    };
    if (q32)
        store(amax, true, q32 + at, scales32 + ((size_t)row * G + g) * 4);
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 8));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 16));
    store(amax, false, q + at, scales + (size_t)row * G + g);
}

// ---- 6. SwiGLU + quantiser: one warp per (route, 128-wide group of I) ------------------
// inter = (g * 1/(1+exp(-g))) * u with gate = columns [0,I), up = [I,2I)
// (kernels/moe.cpp:160-183), then the per-128 quantiser; codes in tensor-operand order.
// one warp: 128 values of one route, written to `group_dst` (the 128 code bytes of the group)
// and `scale_dst`
// a32: one scale per 32 values (scale_dst[0..3], the lane's block is lane / 8) instead of one
// per 128 (scale_dst[0])
__device__ __forceinline__ void swiglu_quant_warp(const float* __restrict__ gate_row,
                                                  const float* __restrict__ up_row, int lane,
                                                  int8_t* group_dst, float* scale_dst,
                                                  bool a32 = false) {
    const float* gp = gate_row + lane * 4;
    const float* up = up_row + lane * 4;
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float gate = gp[i];
        const float e = (float)exp(-(double)gate);
        const float s = __fdiv_rn(1.f, __fadd_rn(1.f, e));
        v[i] = __fmul_rn(__fmul_rn(gate, s), up[i]);
    }
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)  // the lane's 32-block: eight lanes
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    if (!a32) {
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 8));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 16));
    }
    float scale, inv;
    b2w4_quant_params(amax, scale, inv);
    const int c0 = b2w4_quant_code(v[0], inv), c1 = b2w4_quant_code(v[1], inv);
    const int c2 = b2w4_quant_code(v[2], inv), c3 = b2w4_quant_code(v[3], inv);
    if (a32) {
        if ((lane & 7) == 0)
            scale_dst[lane >> 3] = scale;
    } else if (lane == 0) {
        *scale_dst = scale;
    }
    // tensor-operand order inside the group: [word position][even words of the four
    // 32-blocks, then the odd words]; the lane holds k = 4*lane..+3: 32-block lane/8, even
    // codes at even index 2*(lane%8), 2*(lane%8)+1
    int8_t* blk = group_dst + ((lane & 7) >> 1) * 32 + (lane >> 3) * 4 + (lane & 1) * 2;
    *reinterpret_cast<char2*>(blk) = make_char2((signed char)c0, (signed char)c2);
    *reinterpret_cast<char2*>(blk + 16) = make_char2((signed char)c1, (signed char)c3);
}

// scales: [routes][scale_stride].  offsets (null = per-128 everywhere): first compact route of
// every expert, [num_experts + 1]; a route whose expert holds several routes is quantised per
// 32 values (scales[r][4*g + block]), a lone route per 128 (scales[r][g]).
__global__ void moe_swiglu_quant_kernel(const float* __restrict__ gu, int routes,
                                        int intermediate, int8_t* __restrict__ q,
                                        float* __restrict__ scales, int scale_stride,
                                        const int32_t* __restrict__ offsets, int num_experts,
                                        const int32_t* __restrict__ route_lo,
                                        const int32_t* __restrict__ route_hi) {
    b2w4_pdl_chain_entry();
    const int groups = intermediate >> 7;
    const long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)routes * groups)
        return;
    const int r = (int)(wid / groups), g = (int)(wid % groups);
    // expert-parallel runs only own the compact positions of their experts
    if (route_lo && (r < *route_lo || r >= *route_hi))
        return;
    bool a32 = false;
    if (offsets) {  // the expert of compact route r: offsets[e] <= r < offsets[e + 1]
        int lo = 0, hi = num_experts;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (offsets[mid] <= r)
                lo = mid;
            else
                hi = mid;
        }
        a32 = offsets[lo + 1] - offsets[lo] >= 2;
    }
    const float* gp = gu + (size_t)r * 2 * intermediate + (size_t)g * 128;
    swiglu_quant_warp(gp, gp + intermediate, lane,
                      q + (size_t)r * intermediate + (size_t)g * 128,
                      scales + (size_t)r * scale_stride + (a32 ? g * 4 : g), a32);
}

// ---- 8. combine: one block per (token, 512 hidden columns) -------------------------------
// out[t] starts at 0 and takes fma(w, y, out) for the token's experts in ascending id
// (kernels/moe.cpp:642-645, :966, :1100-1110).  The token's k routes are put in that order
// once per block; pos == nullptr reads route rows in (token, route) order.
constexpr int kCombineThreads = 128;
__global__ void __launch_bounds__(kCombineThreads)
moe_combine_kernel(const float* __restrict__ dn, const int32_t* __restrict__ idx,
                   const float* __restrict__ weights, const int32_t* __restrict__ pos,
                   int tokens, int top_k, int hidden_size, float* __restrict__ out, int ldo) {
    b2w4_pdl_chain_entry();
    __shared__ int s_row[kMaxTopK];
    __shared__ float s_w[kMaxTopK];
    const int t = blockIdx.y;
    if (threadIdx.x < top_k) {
        // rank of this route among the token's routes by expert id (ids are distinct, except
        // for the repeated placeholder slots of a degenerate row: ties go to the lower slot)
        const int j = threadIdx.x;
        const int key = idx[(size_t)t * top_k + j];
        // loaded before the rank is known: one memory round trip instead of two
        const int row = pos ? pos[(size_t)t * top_k + j] : t * top_k + j;
        const float w = weights[(size_t)t * top_k + j];
        int rank = 0;
        for (int o = 0; o < top_k; ++o) {
            const int other = idx[(size_t)t * top_k + o];
            rank += other < key || (other == key && o < j);
        }
        s_row[rank] = row;
        s_w[rank] = w;
    }
    __syncthreads();
    const int d = (blockIdx.x * kCombineThreads + threadIdx.x) * 4;
    if (d >= hidden_size)
        return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < top_k; ++j) {
        const float w = s_w[j];
        const float4 y = *reinterpret_cast<const float4*>(dn + (size_t)s_row[j] * hidden_size + d);
        acc.x = __fmaf_rn(w, y.x, acc.x);
        acc.y = __fmaf_rn(w, y.y, acc.y);
        acc.z = __fmaf_rn(w, y.z, acc.z);
        acc.w = __fmaf_rn(w, y.w, acc.w);
    }
    float* o = out + (size_t)t * ldo + d;
    o[0] = acc.x, o[1] = acc.y, o[2] = acc.z, o[3] = acc.w;  // ldo need not be a multiple of 4
}

// ---- expert-parallel hand-over: route outputs in (token, route) order -------------------
// Row t*top_k+j takes the down-projection output of token t's j-th route when that route's
// expert is one of this rank's, zeros otherwise; summed over the ranks (each row has exactly
// one owner, so the sum only adds zeros) the buffer holds every route's output.
__global__ void moe_scatter_routes_kernel(const float* __restrict__ dn,
                                          const int32_t* __restrict__ idx,
                                          const int32_t* __restrict__ pos, int routes,
                                          int hidden_size, int expert_begin, int expert_count,
                                          float* __restrict__ route_out) {
    b2w4_pdl_chain_entry();
    const int r = blockIdx.y;
    const int d = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (r >= routes || d >= hidden_size)
        return;
    const int e = idx[r] - expert_begin;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (e >= 0 && e < expert_count)
        v = *reinterpret_cast<const float4*>(dn + (size_t)pos[r] * hidden_size + d);
    *reinterpret_cast<float4*>(route_out + (size_t)r * hidden_size + d) = v;
}

// ---- expert-parallel hand-over inside the kernels ---------------------------------------
// Instead of a zero-padded buffer summed by an all-reduce call, the owner of a route stores its
// output row into every rank's staging buffer over peer mappings, each value paired with the
// exchange number in one 8-byte word (the same protocol as the tensor-parallel matmul's
// all-gather); rows of other ranks' experts are left to their owners.
__global__ void moe_scatter_routes_peers_kernel(const float* __restrict__ dn,
                                                const int32_t* __restrict__ idx,
                                                const int32_t* __restrict__ pos, int routes,
                                                int hidden_size, int expert_begin,
                                                int expert_count, int stage_rows,
                                                const b2w4_tp_args peers) {
    b2w4_pdl_chain_entry();
    const int r = blockIdx.y;
    const int d = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (r >= routes || d >= hidden_size)
        return;
    const int e = idx[r] - expert_begin;
    if (e < 0 || e >= expert_count)
        return;
    const unsigned exchange =
        *reinterpret_cast<const volatile unsigned*>(peers.stage_peer[peers.rank]) + 1u;
    const float4 v = *reinterpret_cast<const float4*>(dn + (size_t)pos[r] * hidden_size + d);
    const unsigned long long tag = (unsigned long long)exchange << 32;
    const ulonglong2 w01 = make_ulonglong2(tag | __float_as_uint(v.x), tag | __float_as_uint(v.y));
    const ulonglong2 w23 = make_ulonglong2(tag | __float_as_uint(v.z), tag | __float_as_uint(v.w));
    const size_t at = kTpStageHeader + (size_t)(exchange & 1) * stage_rows * hidden_size +
                      (size_t)r * hidden_size + d;
#pragma unroll
    for (int p = 0; p < kTpMaxWorld; ++p)
        if (p < peers.world) {
            ulonglong2* dst = reinterpret_cast<ulonglong2*>(peers.stage_peer[p] + at);
            dst[0] = w01;
            dst[1] = w23;
        }
}

// Combine over the staging buffer: as moe_combine_kernel, but every value is taken from the
// current exchange's half once it carries the exchange number (bounded wait: `wait_limit` SM
// cycles).  The last block advances the count of completed exchanges.  An output that lacks
// one of its rows becomes a quiet NaN, never a sum over stale rows.
__global__ void __launch_bounds__(kCombineThreads)
moe_combine_staged_kernel(unsigned long long* stage, int stage_rows,
                          const int32_t* __restrict__ idx, const float* __restrict__ weights,
                          const int32_t* __restrict__ pos, int tokens, int top_k, int hidden_size,
                          float* __restrict__ out, int ldo, unsigned* done, int* status,
                          unsigned long long wait_limit) {
    b2w4_pdl_chain_entry();
    __shared__ int s_row[kMaxTopK];
    __shared__ float s_w[kMaxTopK];
    const int t = blockIdx.y;
    unsigned* count = reinterpret_cast<unsigned*>(stage);
    const unsigned exchange = *reinterpret_cast<volatile unsigned*>(count) + 1u;
    if (threadIdx.x < top_k) {
        const int j = threadIdx.x;
        const int key = idx[(size_t)t * top_k + j];
        const float w = weights[(size_t)t * top_k + j];
        int rank = 0;
        for (int o = 0; o < top_k; ++o) {
            const int other = idx[(size_t)t * top_k + o];
            rank += other < key || (other == key && o < j);
        }
        // rows in compact order (stored by the down-projection itself) or in (token, route)
        // order (stored by the scatter kernel)
        s_row[rank] = pos ? pos[(size_t)t * top_k + j] : t * top_k + j;
        s_w[rank] = w;
    }
    __syncthreads();
    const int d = (blockIdx.x * kCombineThreads + threadIdx.x) * 4;
    if (d < hidden_size) {
        const unsigned long long* half =
            stage + kTpStageHeader + (size_t)(exchange & 1) * stage_rows * hidden_size;
        const long long t0 = clock64();
        bool gave_up = false;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < top_k; ++j) {
            const volatile unsigned long long* src = half + (size_t)s_row[j] * hidden_size + d;
            unsigned long long w0, w1, w2, w3;
            for (;;) {
                w0 = src[0], w1 = src[1], w2 = src[2], w3 = src[3];
                if (((unsigned)(w0 >> 32) == exchange && (unsigned)(w1 >> 32) == exchange &&
                     (unsigned)(w2 >> 32) == exchange && (unsigned)(w3 >> 32) == exchange) ||
                    gave_up)
                    break;
                if ((unsigned long long)(clock64() - t0) > wait_limit) {
                    b2w4_report_timeout(status);
                    gave_up = true;
                }
            }
            if (gave_up) {
                acc = make_float4(__uint_as_float(0x7FC00000u), __uint_as_float(0x7FC00000u),
                                  __uint_as_float(0x7FC00000u), __uint_as_float(0x7FC00000u));
                break;
            }
            const float w = s_w[j];
            acc.x = __fmaf_rn(w, __uint_as_float((unsigned)w0), acc.x);
            acc.y = __fmaf_rn(w, __uint_as_float((unsigned)w1), acc.y);
            acc.z = __fmaf_rn(w, __uint_as_float((unsigned)w2), acc.z);
            acc.w = __fmaf_rn(w, __uint_as_float((unsigned)w3), acc.w);
        }
        float* o = out + (size_t)t * ldo + d;
        o[0] = acc.x, o[1] = acc.y, o[2] = acc.z, o[3] = acc.w;
    }
    __syncthreads();  // every thread of the block has read the count
    if (threadIdx.x == 0 && atomicAdd(done, 1u) == gridDim.x * gridDim.y - 1) {
        *done = 0;  // ready for the next launch
        *count = exchange;
    }
}

// ---- 5 / 7 (few tokens). grouped expert matmul, decode variant -------------------------
// Used for up to kFusedSwigluTokens tokens, where an expert has one or two routes: items
// (tile pair, group) are spread over all warps, the integer sums go through shared memory and
// a second phase runs the fp32 chains; SwiGLU and its quantiser can run in the prologue.  The
// variant below (register accumulators) is faster from a few routes per expert on; this one
// is faster for a decode step (measured on a Qwen3-30B-shaped layer: 26.9 us against 29.0 us
// per layer for one token, 341 us against 272 us for 256 tokens).
// grid = (CTAs per expert, experts that have routes).  CTA (c, y) owns `tpc` 8-row tiles of
// one expert's slice of the aggregate weight and every route of that expert.  The slice's
// nibble stream is bulk-copied into shared memory once and reused for all of the expert's
// routes, eight at a time: the routes are the eight columns of the warp-level int8 tensor
// instruction (mma.sync m16n8k32), the 16 weight rows of a tile pair its rows.  The math is
// the dense small-batch kernel's: phase 1 integer group sums (a weight word w of 8 nibbles
// splits into signed bytes 16 q, and an accumulator that starts at 0x49400000 ends as the bits of
// the float 786432 + sum: no pass and no barrier for sums of codes; one token, 128 experts of
// 768: 23.2 -> 22.6 us), phase 2 the fp32 chain per (tile, route, weight row) in ascending
// group order.
constexpr int kSW = 8;          // warps
constexpr int kST = kSW * 32;
constexpr int kSR = 8;          // routes per pass
constexpr int kSmallTiles = 16; // tiles per CTA at most
constexpr int kCombineCluster = 8;

struct GroupedSmallArgs {
    const uint8_t* nib;
    const void* scl;
    const int8_t* qa;         // [rows][K] int8, tensor-operand order inside each group
    const float* as;          // [rows][G]
    const float* gate_up;     // if set (few routes): the activations are silu(gate)*up of these
                              // fp32 [routes][2K] rows, quantised here instead of read from qa
    const int4* slots;        // y-th expert with routes: (expert, first route, end), else empty
    // One token, route y is its y-th.  First matmul (kFromLogits): every block picks its own route
    // from the logits (y + 1 rounds), and the first one writes them all.  (The block that selects
    // and compacts in the router kernel waits for the others' logits through a fence and a
    // counter, and this kernel for that block.)  Second matmul (kFromRoutes): idx is read.
    const float* logits;
    int num_experts, top_k;
    int32_t* idx;
    float* weights;
    // One token, second matmul: the routes' blocks of one tile range are a cluster (along x), which
    // combines their rows through distributed shared memory into this row (null: `out` and a
    // combine launch)
    float* combined;
    int expert_begin;         // first expert whose weights this aggregate holds
    int expert_count;         // experts held
    const int32_t* row_map;   // route -> activation row, or null for identity
    float* out;               // [routes][n_e]
    int* status;
    int k, groups, n_e, tiles_e, tpc, d_stride;
    b2w4_tp_args peers;       // world != 0: rows go, tagged, to every rank's staging buffer
    int stage_rows;           // rows per half of that buffer
};

__device__ __forceinline__ void moe_mma_16x8x32(int (&d)[4], uint32_t a0, uint32_t a1,
                                                uint32_t a2, uint32_t a3, uint32_t b0,
                                                uint32_t b1, int4 c) {
    // lane (gid = lane/4, tid = lane%4): a0 row gid, k 4*tid..+3; a1 row gid+8; a2/a3 k+16;
    // b0 k 4*tid..+3 of column gid, b1 k+16; d0/d1 row gid, columns 2*tid, 2*tid+1; d2/d3 row
    // gid+8.
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c.x), "r"(c.y), "r"(c.z),
          "r"(c.w));
}

// Where a block's route comes from: the slot records, the logits, the list of the token's routes.
constexpr int kFromSlots = 0, kFromLogits = 1, kFromRoutes = 2;
template <bool SCL16, int FROM>
__global__ void __launch_bounds__(kST, 2)
moe_grouped_small_kernel(const GroupedSmallArgs a) {
    b2w4_pdl_chain_entry();
    extern __shared__ __align__(128) uint8_t smem[];
    // blockIdx.y walks the experts that have routes, not all experts: a decode token
    // touches top_k of them
    const bool combined = FROM == kFromRoutes && a.combined;
    const int y = combined ? blockIdx.x : blockIdx.y, x = combined ? blockIdx.y : blockIdx.x;
    int4 slot = make_int4(0, y, y + 1, 0);
    if (FROM == kFromSlots) {
        slot = a.slots[y];
    } else if (FROM == kFromLogits) {
        // by every warp: no barrier before the weights are asked for
        float logit;
        const int picked =
            pick_routes_any(a.logits, a.num_experts, y + 1, threadIdx.x & 31, logit);
        slot.x = __shfl_sync(0xffffffffu, picked, y);
    } else {
        slot.x = a.idx[y];
    }
    const int e_all = slot.x, r0 = slot.y, r1 = slot.z;
    const int e = e_all - a.expert_begin;  // index inside the aggregate held here
    if (e < 0 || e >= a.expert_count)
        return;
    const int tl0 = x * a.tpc;
    const int ntile = min(a.tpc, a.tiles_e - tl0);
    if (r0 >= r1 || ntile <= 0)
        return;
    const int G = a.groups, K = a.k;
    const int tile_bytes = G * 512;
    const int scl_tile_bytes = G * 8 * (SCL16 ? 2 : 4);
    uint8_t* s_w = smem;
    uint8_t* s_scl = s_w + (size_t)a.tpc * tile_bytes;
    uint4* s_qa = reinterpret_cast<uint4*>(s_scl + (size_t)a.tpc * scl_tile_bytes);  // [kSR][K]
    float* s_as = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(s_qa) + (size_t)kSR * K);
    float* s_d = s_as + kSR * G;  // [tpc][G][kSR][8] + pad
    uint64_t* s_bar = reinterpret_cast<uint64_t*>(
        (reinterpret_cast<uintptr_t>(s_d + (size_t)a.tpc * a.d_stride) + 7) & ~uintptr_t(7));

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tid = lane & 3;
    const size_t gtile0 = (size_t)e * a.tiles_e + tl0;  // tile index in the aggregate

    if (warp == 0) {
        if (lane == 0)
            mbar_init(&s_bar[0], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
            const uint32_t wb = (uint32_t)ntile * tile_bytes, sb = (uint32_t)ntile * scl_tile_bytes;
            mbar_expect_tx(&s_bar[0], wb + sb);
            bulk_g2s(s_w, a.nib + gtile0 * tile_bytes, wb, &s_bar[0]);
            bulk_g2s(s_scl, reinterpret_cast<const uint8_t*>(a.scl) + gtile0 * scl_tile_bytes, sb,
                     &s_bar[0]);
        }
    }
    __syncthreads();  // no warp polls the barrier word before it is one
    if (FROM == kFromLogits && x == 0 && y == 0 && warp == kSW - 1)
        select_routes_any(a.logits, 0, a.num_experts, a.top_k, a.idx, a.weights, lane);
    __shared__ float s_row[FROM == kFromRoutes ? kSmallTiles * 8 : 1];  // this route's rows
    const int npair = (ntile + 1) >> 1;
    const int n_items = npair * G;
    const uint32_t* s_w32 = reinterpret_cast<const uint32_t*>(s_w);
    const int tile_words = tile_bytes >> 2;
    bool weights_ready = false;

    for (int base = r0; base < r1; base += kSR) {
        const int mc = min(kSR, r1 - base);
        // quantised activations of this pass's routes
        if (a.gate_up) {
            // every CTA of the expert repeats this for the expert's routes: cheap for the few
            // routes of a decode step, and it saves a launch
            for (int task = warp; task < mc * G; task += kSW) {
                const int mi = task / G, g = task - mi * G;
                const float* gp = a.gate_up + (size_t)(base + mi) * 2 * K + (size_t)g * 128;
                swiglu_quant_warp(gp, gp + K, lane,
                                  reinterpret_cast<int8_t*>(s_qa) + (size_t)mi * K + (size_t)g * 128,
                                  s_as + mi * G + g);
            }
        } else {
            for (int i = threadIdx.x; i < mc * (K / 16); i += kST) {
                const int mi = i / (K / 16), c = i - mi * (K / 16);
                const int src_row = FROM == kFromLogits ? 0 : a.row_map ? a.row_map[base + mi] : base + mi;
                s_qa[mi * (K / 16) + c] =
                    reinterpret_cast<const uint4*>(a.qa + (size_t)src_row * K)[c];
            }
            for (int i = threadIdx.x; i < mc * G; i += kST) {
                const int mi = i / G, g = i - mi * G;
                const int src_row = FROM == kFromLogits ? 0 : a.row_map ? a.row_map[base + mi] : base + mi;
                s_as[mi * G + g] = a.as[(size_t)src_row * G + g];
            }
        }
        if (!weights_ready) {
            if (!mbar_wait_bounded(&s_bar[0])) {
                if (lane == 0)
                    b2w4_report_timeout(a.status);
                // The status word says that the rows are void.  In a cluster the warp goes on with
                // what is there, to both of its barriers: the other blocks read this one's rows.
                if (!combined)
                    return;
            }
            weights_ready = true;
        }
        __syncthreads();
        // phase 1: item = (pair of tiles = 16 weight rows, group); columns = routes
        const int bcol = gid < mc ? gid : 0;  // unused columns repeat route 0, never read back
        const int qa_base = bcol * (K >> 4) + tid * 2;
#pragma unroll 2
        for (int it = warp; it < n_items; it += kSW) {
            const int tp = it / G;
            const int g = it - tp * G;
            const int t0 = tp * 2;
            const bool two = t0 + 1 < ntile;
            // word `lane` of the 128 bytes of (tile, group, 32-block s): row gid, k 8*tid..+7
            const int wbase = t0 * tile_words + g * 128 + lane;
            uint32_t lo0[4], hi0[4], lo1[4], hi1[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const uint32_t u = s_w32[wbase + s * 32];
                const uint32_t v = two ? s_w32[wbase + tile_words + s * 32] : 0u;  // q = 0
                lo0[s] = (u << 4) & 0xF0F0F0F0u;
                hi0[s] = u & 0xF0F0F0F0u;
                lo1[s] = (v << 4) & 0xF0F0F0F0u;
                hi1[s] = v & 0xF0F0F0F0u;
            }
            const uint4 be = s_qa[qa_base + g * 8], bo = s_qa[qa_base + g * 8 + 1];
            // two chains of two instructions (latency), joined by one add
            const int4 start = make_int4(0x49400000, 0x49400000, 0x49400000, 0x49400000);
            auto value = [](int d) { return __fsub_rn(__int_as_float(d), 786432.f); };
            int d[4], e2[4];
            moe_mma_16x8x32(d, lo0[0], lo1[0], lo0[1], lo1[1], be.x, be.y, start);
            moe_mma_16x8x32(e2, hi0[0], hi1[0], hi0[1], hi1[1], bo.x, bo.y, make_int4(0, 0, 0, 0));
            moe_mma_16x8x32(d, lo0[2], lo1[2], lo0[3], lo1[3], be.z, be.w,
                            make_int4(d[0], d[1], d[2], d[3]));
            moe_mma_16x8x32(e2, hi0[2], hi1[2], hi0[3], hi1[3], bo.z, bo.w,
                            make_int4(e2[0], e2[1], e2[2], e2[3]));
            const int dbase = t0 * a.d_stride + g * (kSR * 8) + gid;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int mi = tid * 2 + c;
                if (mi < mc) {
                    s_d[dbase + mi * 8] = value(d[c] + e2[c]);
                    if (two)
                        s_d[dbase + a.d_stride + mi * 8] = value(d[2 + c] + e2[2 + c]);
                }
            }
        }
        __syncthreads();
        // phase 2
#pragma unroll 1
        for (int t = threadIdx.x; t < ntile * kSR * 8; t += kST) {
            const int rr = t & 7, mi = (t >> 3) % kSR, tl = t / (8 * kSR);
            if (mi >= mc)
                continue;
            const float* dsrc = s_d + tl * a.d_stride + mi * 8 + rr;
            const float* as = s_as + mi * G;
            float acc = 0.f;
#pragma unroll 4
            for (int g = 0; g < G; ++g) {
                const float ws =
                    SCL16 ? __half2float(
                                reinterpret_cast<const __half*>(s_scl)[(tl * G + g) * 8 + rr])
                          : reinterpret_cast<const float*>(s_scl)[(tl * G + g) * 8 + rr];
                acc = __fmaf_rn(dsrc[g * kSR * 8], __fmul_rn(ws, as[g]), acc);
            }
            const int n = (tl0 + tl) * 8 + rr;
            if (combined) {
                s_row[tl * 8 + rr] = acc;
            } else if (n < a.n_e) {
                if (a.peers.world == 0) {
                    a.out[(size_t)(base + mi) * a.n_e + n] = acc;
                } else {
                    // expert-parallel hand-over: the row (its compact position is the same
                    // on every rank) goes to every rank's staging buffer, each value tagged
                    // with the exchange number in one 8-byte word
                    const unsigned exchange =
                        *reinterpret_cast<const volatile unsigned*>(
                            a.peers.stage_peer[a.peers.rank]) + 1u;
                    const unsigned long long word =
                        ((unsigned long long)exchange << 32) | __float_as_uint(acc);
                    const size_t at = kTpStageHeader +
                                      (size_t)(exchange & 1) * a.stage_rows * a.n_e +
                                      (size_t)(base + mi) * a.n_e + n;
#pragma unroll
                    for (int p = 0; p < kTpMaxWorld; ++p)
                        if (p < a.peers.world)
                            a.peers.stage_peer[p][at] = word;
                }
            }
        }
        __syncthreads();
    }
    if (combined) {
        // moe_combine_kernel's sum over the routes in ascending expert id, each block its share of
        // the tile range's rows
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        const int routes = gridDim.x;
        __shared__ int s_from[kCombineCluster];
        __shared__ float s_weight[kCombineCluster];
        if ((int)threadIdx.x < routes) {
            const int j = threadIdx.x, key = a.idx[j];
            int rank = 0;
            for (int o = 0; o < routes; ++o) {
                const int other = a.idx[o];
                rank += other < key || (other == key && o < j);
            }
            s_from[rank] = j;
            s_weight[rank] = a.weights[j];
        }
        cluster.sync();  // every route's rows, and the order
        const int rows = min(ntile * 8, a.n_e - tl0 * 8);
        for (int i = y * kST + threadIdx.x; i < rows; i += routes * kST) {
            float acc = 0.f;
            for (int j = 0; j < routes; ++j)
                acc = __fmaf_rn(s_weight[j], cluster.map_shared_rank(s_row, s_from[j])[i], acc);
            a.combined[tl0 * 8 + i] = acc;
        }
        cluster.sync();  // nobody leaves while its rows may still be read
    }
}

int grouped_small_d_stride(int groups) { return groups * kSR * 8 + 8; }

size_t grouped_small_smem(int k, int groups, int tpc, bool scl16) {
    return (size_t)tpc * groups * 512 + (size_t)tpc * groups * 8 * (scl16 ? 2 : 4) +
           (size_t)kSR * k + sizeof(float) * kSR * groups +
           sizeof(float) * (size_t)tpc * grouped_small_d_stride(groups) + 8 + 16;
}

// ---- 5 / 7. grouped expert matmul over ragged route lists ------------------------------
// Work: an expert's routes, sixteen at a time (a pass), against its tile pairs (16 weight rows
// each).  A unit is one pass against a pair per warp of a CTA; the units of all experts lie in
// one line (expert, pass, pairs) of which every CTA takes an equal, contiguous share, two CTAs
// of eight warps per SM, so that one computes while the other changes to another pass, or one
// CTA of sixteen warps where a pass's rows leave no room for two.  A pass's int8 rows and scales
// are staged in shared memory once and serve all units of the share that belong to it.
//
// The integer sums come from the warp-level int8 tensor instruction (mma.sync m16n8k32): the
// pair's weight rows are its rows, eight routes its columns.  A warp runs the whole K loop of its
// pair on its own: the pair's weights stream through a ring in shared memory that only this warp
// reads and fills (cp.async), kDepth - 1 groups ahead, on into the next pair, with no barrier in
// the K loop.  (Straight into registers, three groups ahead, they came later: a warp's
// outstanding loads share six scoreboards, so a wait for an old group waited for the newest
// too.)
//
// A word is split into signed bytes 16 q (lo = (w << 4) & 0xF0F0F0F0 for even k, hi = w &
// 0xF0F0F0F0 for odd k: a nibble in the upper half of a byte is its two's complement value times
// sixteen).  Every accumulator starts at 0x49400000, the bits of the float 786432 whose last place
// is worth 1/16, and ends as 0x49400000 + 16 D: the bits of 786432 + D, exactly, since
// |16 D| <= 128 * 127 * 128 < 2^22.  So D costs one subtraction, for two columns at once, and no
// correction by the sum of the codes has to be made, staged and read (with unsigned q + 8 bytes it
// had: 128-bit reads of four words per instruction were most of the shared-memory traffic, whose
// pipe was 68 % busy; 256 tokens, 128 experts of 768: 231 -> 191 us).  D is folded into fp32 chain values
// y = fma(float(D), fp32(ws*as), y)  that stay in the warp's registers until the last group, two
// columns per instruction.  The math is the dense kernels', route by route.
// What bounds it: nothing alone.  256 tokens over 128 experts of 768, gate_up / down: 0.10 / 0.06
// ms, about three times what the weights take from HBM (36 / 27 % of its rate), issue slots 62 /
// 61 % busy, the shared-memory pipe 57 / 54 %; a warp waits 5.8 cycles per instruction with 3.6
// warps per scheduler (1.5 for the result before it, 1.1 for its turn, 0.8 for the fp32 pipe, 0.6
// for shared memory).  Experts with more than sixteen routes stream and split their weights again.
constexpr int kGR = 16;         // routes per pass: two column blocks
constexpr int kRowPad = 16;     // bytes added to a staged activation row: conflict-free reads

struct GroupedArgs {
    const uint8_t* nib;
    const void* scl;
    const int8_t* qa;         // [rows][K] int8, tensor-operand order inside each group
    const float* as;          // [rows][as_stride]: one scale per 128 values at [g]
    // The reference's rule for an expert that holds SEVERAL rows (kernels/moe.cpp:1055-1058
    // -> kernels/matmul_w4.cpp:1125-1154): one activation scale per 32 values.  qa32 / as32 are
    // those rows quantised that way (as32[r][4*g + block]); null = per-128 for every expert.
    // An expert with a single row keeps the per-128 rule (:1058-1075).
    const int8_t* qa32;
    const float* as32;
    int as_stride, as32_stride;
    const int4* slots;        // y-th expert with routes: (expert, first route, end), else empty
    int slot_count;           // entries of slots that can hold an expert
    int expert_begin;         // first expert whose weights this aggregate holds
    int expert_count;         // experts held
    const int32_t* row_map;   // route -> activation row, or null for identity
    float* out;               // [routes][n_e]
    int k, groups, n_e, tiles_e;
};

template <int BYTES>
__device__ __forceinline__ void moe_cp_async(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "n"(BYTES)
                 : "memory");
}

// one group's weights of a lane: a word of each 32-k block of both tiles' row gid, both scales
struct PairWords {
    uint32_t w[2][4];
    float ws[2];
};
// a warp's ring slot: [2 tiles][512 B], then [2 tiles][8 scales]
template <bool SCL16>
constexpr int kPairSlot = 1024 + (SCL16 ? 32 : 64);

// Folds one group of sixteen weight rows into the chain values of `ncb` blocks of eight routes.
// acc[j][0]: row gid, routes 2*tid and 2*tid+1 of block j; acc[j][1]: row gid+8.
template <bool A32>
__device__ __forceinline__ void pair_group(const PairWords& pw, const uint8_t* rows,
                                           int row_bytes, const float* s_as, int g, int ncb,
                                           int tid, uint64_t (&acc)[2][2]) {
    uint32_t lo[2][4], hi[2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            lo[t][b] = (pw.w[t][b] << 4) & 0xF0F0F0F0u;
            hi[t][b] = pw.w[t][b] & 0xF0F0F0F0u;
        }
    const uint64_t magic = b2w4_pack2(786432.f, 786432.f);
    const int4 start = make_int4(0x49400000, 0x49400000, 0x49400000, 0x49400000);
    const uint64_t w0 = b2w4_pack2(pw.ws[0], pw.ws[0]), w1 = b2w4_pack2(pw.ws[1], pw.ws[1]);
    auto fold = [&](const int (&c)[4], uint64_t as2, uint64_t (&y)[2]) {
        // c = 0x49400000 + 16 D: as a float 786432 + D, exactly
        const uint64_t d0 = b2w4_sub2(b2w4_pack2(__int_as_float(c[0]), __int_as_float(c[1])), magic);
        const uint64_t d1 = b2w4_sub2(b2w4_pack2(__int_as_float(c[2]), __int_as_float(c[3])), magic);
        y[0] = b2w4_fma2(d0, b2w4_mul2(w0, as2), y[0]);
        y[1] = b2w4_fma2(d1, b2w4_mul2(w1, as2), y[1]);
    };
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        if (j < ncb) {  // warp-uniform; unused columns of the last block are never stored
            const uint4* bp = reinterpret_cast<const uint4*>(rows + j * 8 * row_bytes + g * 128);
            const uint4 be = bp[0], bo = bp[1];
            const uint32_t bev[4] = {be.x, be.y, be.z, be.w}, bov[4] = {bo.x, bo.y, bo.z, bo.w};
            if (A32) {
                // one instruction = one 32-block: its own accumulator and activation scale,
                // folded in ascending block order (kernels/matmul_w4.cpp:785-901)
                const ulonglong2* ap =
                    reinterpret_cast<const ulonglong2*>(s_as) + (g * (kGR / 2) + j * 4 + tid) * 2;
                const ulonglong2 a01 = ap[0], a23 = ap[1];
                const uint64_t as2[4] = {a01.x, a01.y, a23.x, a23.y};
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    int c[4];
                    moe_mma_16x8x32(c, lo[0][b], lo[1][b], hi[0][b], hi[1][b], bev[b], bov[b],
                                    start);
                    fold(c, as2[b], acc[j]);
                }
            } else {
                // two chains of two instructions (latency), joined by one add
                const int at = g * (kGR / 2) + j * 4 + tid;
                int c[4], c2[4];
                moe_mma_16x8x32(c, lo[0][0], lo[1][0], hi[0][0], hi[1][0], bev[0], bov[0],
                                start);
                moe_mma_16x8x32(c2, lo[0][1], lo[1][1], hi[0][1], hi[1][1], bev[1], bov[1],
                                make_int4(0, 0, 0, 0));
                moe_mma_16x8x32(c, lo[0][2], lo[1][2], hi[0][2], hi[1][2], bev[2], bov[2],
                                make_int4(c[0], c[1], c[2], c[3]));
                moe_mma_16x8x32(c2, lo[0][3], lo[1][3], hi[0][3], hi[1][3], bev[3], bov[3],
                                make_int4(c2[0], c2[1], c2[2], c2[3]));
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    c[i] += c2[i];
                fold(c, reinterpret_cast<const uint64_t*>(s_as)[at], acc[j]);
            }
        }
    }
}

template <bool SCL16, int kGW, int kDepth>
__global__ void __launch_bounds__(kGW * 32, 16 / kGW)
moe_grouped_gemv_kernel(const GroupedArgs a) {
    b2w4_pdl_chain_entry();
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int kSlot = kPairSlot<SCL16>;
    const int G = a.groups, K = a.k;
    const int row_bytes = K + kRowPad;
    // activation scales [G][kGR], per 32 values [G][kGR / 2][4 blocks][2 routes]
    float* s_as = reinterpret_cast<float*>(smem);
    uint8_t* s_qa = reinterpret_cast<uint8_t*>(s_as + (size_t)4 * G * kGR);       // [kGR][K+pad]
    uint8_t* s_ring = s_qa + (size_t)kGR * row_bytes;                             // [kGW][kDepth]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tid = lane & 3;

    // Passes before a slot (experts held elsewhere have none), by every warp for itself: a lane
    // sums `per` slots in a row, the warp the lanes.  One trip to L2 and no barrier before the
    // first weights are asked for, which is what a few routes wait for.
    const int per = (a.slot_count + 31) / 32;
    auto passes_of = [&](int4 slot) {
        const int e = slot.x - a.expert_begin;
        return e >= 0 && e < a.expert_count && slot.z > slot.y
                   ? (slot.z - slot.y + kGR - 1) / kGR
                   : 0;
    };
    auto scan = [&](int v) {  // inclusive, over the lanes
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int other = __shfl_up_sync(0xffffffffu, v, off);
            if (lane >= off)
                v += other;
        }
        return v;
    };
    int4 own = make_int4(0, 0, 0, 0);
    int mine = 0;
    for (int i = 0; i < per; ++i)
        if (lane * per + i < a.slot_count) {
            own = a.slots[lane * per + i];
            mine += passes_of(own);
        }
    const int run = scan(mine), before = run - mine;
    // the slot that pass p belongs to, and p's number within it
    auto find = [&](int p, int4& slot) {
        int at = __popc(__ballot_sync(0xffffffffu, run <= p));  // the lane
        int pre = __shfl_sync(0xffffffffu, before, at);
        int4 mem = own;
        if (per > 1) {
            const int y = at * per + lane;
            mem = lane < per && y < a.slot_count ? a.slots[y] : make_int4(0, 0, 0, 0);
            const int n = passes_of(mem), upto = scan(n);
            at = __popc(__ballot_sync(0xffffffffu, pre + upto <= p));
            pre += __shfl_sync(0xffffffffu, upto - n, at);
        }
        slot.x = __shfl_sync(0xffffffffu, mem.x, at);
        slot.y = __shfl_sync(0xffffffffu, mem.y, at);
        slot.z = __shfl_sync(0xffffffffu, mem.z, at);
        return p - pre;
    };
    const int pairs = a.tiles_e / 2;  // n_e is a multiple of 128
    const int rounds = (pairs + kGW - 1) / kGW;
    const long long total = (long long)__shfl_sync(0xffffffffu, run, 31) * rounds;
    long long u = total * blockIdx.x / gridDim.x;
    const long long u_end = total * (blockIdx.x + 1) / gridDim.x;
    const size_t tile_bytes = (size_t)G * 512, scl_tile_bytes = (size_t)G * (SCL16 ? 16 : 32);

    while (u < u_end) {
        const int pass_all = (int)(u / rounds);
        const int round0 = (int)(u - (long long)pass_all * rounds);
        const int round1 = (int)min((long long)rounds, round0 + (u_end - u));
        u += round1 - round0;
        int4 slot;
        const int pass = find(pass_all, slot);
        const int base = slot.y + pass * kGR;
        const int mc = min(kGR, slot.z - base);
        // the expert's rule: per 32 values when it holds several rows
        const bool a32 = a.qa32 != nullptr && slot.z - slot.y >= 2;
        const int spg = a32 ? 4 : 1;  // scales per group

        // this warp's pairs in the share, group by group: the next one to fetch
        const size_t tile0 = (size_t)(slot.x - a.expert_begin) * a.tiles_e;
        int f_pair = round0 * kGW + warp, f_g = 0, f_slot = 0;
        const int pair_end = min(pairs, round1 * kGW);
        uint8_t* const ring = s_ring + warp * (kDepth * kSlot);
        auto fetch = [&]() {
            if (f_pair < pair_end) {
                const size_t at = (tile0 + 2 * f_pair) * G + f_g;
                uint8_t* dst = ring + f_slot * kSlot;
#pragma unroll
                for (int t = 0; t < 2; ++t)
                    moe_cp_async<16>(dst + t * 512 + lane * 16,
                                     a.nib + (at + (size_t)t * G) * 512 + lane * 16);
                constexpr int kScl = SCL16 ? 16 : 32;  // bytes of a tile's eight scales
                if (lane < kScl / 8) {
                    const int t = lane / (kScl / 16), c = lane % (kScl / 16);
                    moe_cp_async<16>(dst + 1024 + lane * 16,
                                     reinterpret_cast<const uint8_t*>(a.scl) +
                                         (at + (size_t)t * G) * kScl + c * 16);
                }
                f_slot = f_slot + 1 == kDepth ? 0 : f_slot + 1;
                if (++f_g == G) {
                    f_g = 0;
                    f_pair += kGW;
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int i = 0; i < kDepth - 1; ++i)
            fetch();

        // the pass's rows, a warp per row, all copies in flight at once
        for (int mi = warp; mi < mc; mi += kGW) {
            const int row = a.row_map ? a.row_map[base + mi] : base + mi;
            const int8_t* src = (a32 ? a.qa32 : a.qa) + (size_t)row * K;
            const size_t at = (size_t)row * (a32 ? a.as32_stride : a.as_stride);
            const float* as = (a32 ? a.as32 : a.as) + at;
#pragma unroll 4
            for (int c = lane * 16; c < K; c += 32 * 16)
                moe_cp_async<16>(s_qa + (size_t)mi * row_bytes + c, src + c);
            for (int gs = lane; gs < G * spg; gs += 32) {
                const int to = a32 ? (gs >> 2) * (4 * kGR) + (mi >> 1) * 8 + (gs & 3) * 2 + (mi & 1)
                                   : gs * kGR + mi;
                moe_cp_async<4>(s_as + to, as + gs);
            }
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        __syncthreads();

        const int ncb = (mc + 7) >> 3;  // column blocks in this pass: 1 or 2
        const uint8_t* rows = s_qa + gid * row_bytes + tid * 32;
        int slot_at = 0;
#pragma unroll 1
        for (int round = round0; round < round1; ++round) {
            if (round * kGW + warp >= pairs)
                break;
            uint64_t acc[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
            auto run = [&](auto rule) {
#pragma unroll 2
                for (int g = 0; g < G; ++g) {
                    __syncwarp();  // every lane has read the slot that is filled now
                    fetch();
                    asm volatile("cp.async.wait_group %0;" ::"n"(kDepth - 1) : "memory");
                    __syncwarp();
                    const uint8_t* src = ring + slot_at * kSlot;
                    slot_at = slot_at + 1 == kDepth ? 0 : slot_at + 1;
                    PairWords now;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
#pragma unroll
                        for (int b = 0; b < 4; ++b)
                            now.w[t][b] = *reinterpret_cast<const uint32_t*>(src + t * 512 +
                                                                             b * 128 + lane * 4);
                        now.ws[t] =
                            SCL16 ? __half2float(reinterpret_cast<const __half*>(src + 1024)[t * 8 +
                                                                                             gid])
                                  : reinterpret_cast<const float*>(src + 1024)[t * 8 + gid];
                    }
                    pair_group<decltype(rule)::value>(now, rows, row_bytes, s_as, g, ncb, tid,
                                                      acc);
                }
            };
            if (a32)
                run(std::true_type{});
            else
                run(std::false_type{});
            // out[route][n]: the eight lanes of a quarter-warp hold eight consecutive n
            const int n0 = (round * kGW + warp) * 16 + gid;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                float v[2][2];
                b2w4_unpack2(acc[j][0], v[0][0], v[0][1]);
                b2w4_unpack2(acc[j][1], v[1][0], v[1][1]);
#pragma unroll
                for (int cc = 0; cc < 2; ++cc) {
                    const int mi = j * 8 + tid * 2 + cc;
                    if (mi < mc) {
                        float* o = a.out + (size_t)(base + mi) * a.n_e + n0;
                        o[0] = v[0][cc];
                        o[8] = v[1][cc];
                    }
                }
            }
        }
        __syncthreads();  // the staged rows are overwritten by the next pass
    }
}

size_t grouped_smem(int k, int groups, bool scl16, int warps, int depth) {
    return sizeof(float) * kGR * groups * 4 + (size_t)kGR * (k + kRowPad) +
           (size_t)warps * depth * (scl16 ? kPairSlot<true> : kPairSlot<false>);
}

template <int W, int D>
int launch_grouped_as(b2w4_ctx* ctx, const GroupedArgs& a, bool scl16, size_t smem, int routes) {
    auto kern = scl16 ? moe_grouped_gemv_kernel<true, W, D> : moe_grouped_gemv_kernel<false, W, D>;
    static b2w4_smem_optin configured[2];  // per instantiation and device
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, configured[scl16]));
    // no more CTAs than there can be units (a pass holds at least one route)
    const long long units = (long long)routes * ((a.tiles_e / 2 + W - 1) / W);
    const long long room = 16 / W * ctx->sm_count;
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, dim3((int)(units < room ? units : room)),
                                       dim3(W * 32), smem, ctx->stream, a));
    ctx->launches++;
    return B2W4_OK;
}

// Tiles per CTA of the few-token kernel.
int small_tiles(const b2w4_weight* w) {
    int tpc = kSmallTiles;
    while (tpc > 2 &&
           grouped_small_smem(w->k, w->groups, tpc, w->scales_fp16 != 0) > 113 * 1024)
        tpc -= 2;  // even: tiles are taken in pairs
    return tpc;
}

// The routes of a single token; logits null: read from idx.
struct TokenRoutes {
    const float* logits;
    int32_t* idx;
    float* weights;
    float* combined;  // GroupedSmallArgs
};

// `decode` (few tokens): the shared-memory variant, optionally with SwiGLU + quantiser fused
// into its prologue (fused_gate_up = the gate_up matmul's fp32 output).
// qa32 / as32: the same rows quantised per 32 values, for experts that hold several routes
// (null: per-128 for all); as_stride / as32_stride: scales per row of as / as32.
int launch_grouped(b2w4_ctx* ctx, const b2w4_weight* w, int num_experts_all, int expert_begin,
                   int expert_count, int routes, const int8_t* qa, const float* as,
                   int as_stride, const int8_t* qa32, const float* as32, int as32_stride,
                   const int4* slots, const int32_t* row_map, float* out, bool decode,
                   const float* fused_gate_up = nullptr, const b2w4_tp_args* peers = nullptr,
                   int stage_rows = 0, const TokenRoutes* token = nullptr) {
    const int n_e = w->n / expert_count;
    const bool scl16 = w->scales_fp16 != 0;
    const int slots_y = routes < num_experts_all ? routes : num_experts_all;  // grid.y
    if (decode) {
        GroupedSmallArgs a = {};
        a.nib = reinterpret_cast<const uint8_t*>(w->nib);
        a.scl = w->scl;
        a.qa = qa;
        a.as = as;
        a.slots = slots;
        if (token) {
            a.logits = token->logits;
            a.num_experts = num_experts_all;
            a.top_k = routes;
            a.idx = token->idx;
            a.weights = token->weights;
            a.combined = token->combined;
        }
        a.gate_up = fused_gate_up;
        a.expert_begin = expert_begin;
        a.expert_count = expert_count;
        a.row_map = row_map;
        a.out = out;
        a.status = ctx->status_dev;
        if (peers) {
            a.peers = *peers;
            a.stage_rows = stage_rows;
        }
        a.k = w->k;
        a.groups = w->groups;
        a.n_e = n_e;
        a.tiles_e = n_e / 8;
        const int tpc = small_tiles(w);
        a.tpc = tpc;
        a.d_stride = grouped_small_d_stride(w->groups);
        const size_t smem = grouped_small_smem(w->k, w->groups, tpc, scl16);
        if (w->k > (scl16 ? 10752 : 10624))  // the limit of the operator
            return b2w4_fail(ctx, B2W4_E_INVALID, "moe: K=%d needs %zu B shared memory", w->k,
                             smem);
        const int from = !token ? kFromSlots : token->logits ? kFromLogits : kFromRoutes;
        auto kern = from == kFromSlots ? (scl16 ? moe_grouped_small_kernel<true, kFromSlots>
                                                : moe_grouped_small_kernel<false, kFromSlots>)
                    : from == kFromLogits ? (scl16 ? moe_grouped_small_kernel<true, kFromLogits>
                                                   : moe_grouped_small_kernel<false, kFromLogits>)
                                          : (scl16 ? moe_grouped_small_kernel<true, kFromRoutes>
                                                   : moe_grouped_small_kernel<false, kFromRoutes>);
        static b2w4_smem_optin configured[6];  // per instantiation and device
        B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, configured[from * 2 + scl16]));
        const int ranges = (a.tiles_e + tpc - 1) / tpc;
        if (a.combined)
            B2W4_CUDA(ctx, b2w4_launch_chained_cluster(ctx->pdl, kern, dim3(slots_y, ranges),
                                                       dim3(kST), slots_y, smem, ctx->stream, a));
        else
            B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, dim3(ranges, slots_y), dim3(kST),
                                               smem, ctx->stream, a));
        ctx->launches++;
        return B2W4_OK;
    }
    GroupedArgs a = {};
    a.nib = reinterpret_cast<const uint8_t*>(w->nib);
    a.scl = w->scl;
    a.qa = qa;
    a.as = as;
    a.as_stride = as_stride;
    a.qa32 = qa32;
    a.as32 = as32;
    a.as32_stride = as32_stride;
    a.slots = slots;
    a.slot_count = slots_y;
    a.expert_begin = expert_begin;
    a.expert_count = expert_count;
    a.row_map = row_map;
    a.out = out;
    a.k = w->k;
    a.groups = w->groups;
    a.n_e = n_e;
    a.tiles_e = n_e / 8;
    if (w->k > (scl16 ? 7936 : 7808))  // the limit of the operator
        return b2w4_fail(ctx, B2W4_E_INVALID, "moe: K=%d needs too much shared memory", w->k);
    auto bytes = [&](int warps, int depth) {
        return grouped_smem(w->k, w->groups, scl16, warps, depth);
    };
    // two CTAs per SM, else sixteen warps in one, else what the rows leave room for
    if (bytes(8, 6) <= 112 * 1024)
        return launch_grouped_as<8, 6>(ctx, a, scl16, bytes(8, 6), routes);
    if (bytes(16, 6) <= 226 * 1024)
        return launch_grouped_as<16, 6>(ctx, a, scl16, bytes(16, 6), routes);
    return launch_grouped_as<8, 4>(ctx, a, scl16, bytes(8, 4), routes);
}

}  // namespace

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

extern "C" {

int b2w4_moe_select_routes(b2w4_ctx* ctx, const float* logits_dev, int tokens,
                           int num_experts, int top_k, int32_t* indices_dev,
                           float* weights_dev) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!logits_dev || !indices_dev || !weights_dev || tokens <= 0 || num_experts <= 0 ||
        top_k <= 0 || top_k > num_experts || top_k > kMaxTopK ||
        num_experts > kSelectMaxExperts)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "select_routes: need 0 < top_k <= min(experts, %d), experts <= %d "
                         "(tokens=%d experts=%d top_k=%d)", kMaxTopK, kSelectMaxExperts, tokens,
                         num_experts, top_k);
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_select_routes_kernel, dim3((tokens + 3) / 4),
                                       dim3(128), 0, ctx->stream, logits_dev, tokens,
                                       num_experts, top_k, indices_dev, weights_dev));
    ctx->launches++;
    B2W4_CUDA(ctx, cudaGetLastError());
    return B2W4_OK;
}

}  // extern "C"

// The whole MoE op.  With route_out == nullptr it computes every expert and combines into
// out_dev.  With route_out set it is one rank of an expert-parallel group: routing runs over
// all num_experts (replicated), the aggregates hold experts [expert_begin, expert_begin +
// expert_count) only, and the rank's route outputs go to route_out in (token, route) order.
static int moe_run(b2w4_ctx* ctx, const float* hidden_dev, int ldx, int tokens, int hidden_size,
                   const void* router_fp16_dev, int num_experts, int top_k, int intermediate,
                   const b2w4_weight* gate_up, const b2w4_weight* down, int expert_begin,
                   int expert_count, float* out_dev, int ldo, float* route_out,
                   float* logits_dev, int32_t* indices_dev, float* weights_dev,
                   const b2w4_tp_args* peers = nullptr, int stage_rows = 0) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!hidden_dev || !router_fp16_dev || !gate_up || !down || (!out_dev && !route_out))
        return b2w4_fail(ctx, B2W4_E_INVALID, "moe: null argument");
    if (tokens <= 0 || num_experts <= 0 || num_experts > kSelectMaxExperts || top_k <= 0 ||
        top_k > num_experts || top_k > kMaxTopK || hidden_size % 128 || intermediate % 128 || ldx < hidden_size ||
        (out_dev && ldo < hidden_size))
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "moe: bad shape tokens=%d hidden=%d experts=%d top_k=%d inter=%d",
                         tokens, hidden_size, num_experts, top_k, intermediate);
    if (expert_begin < 0 || expert_count <= 0 || expert_begin + expert_count > num_experts)
        return b2w4_fail(ctx, B2W4_E_INVALID, "moe: experts [%d, %d) outside [0, %d)",
                         expert_begin, expert_begin + expert_count, num_experts);
    if (gate_up->k != hidden_size || gate_up->n != expert_count * 2 * intermediate ||
        down->k != intermediate || down->n != expert_count * hidden_size)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "moe: expert aggregates must be gate_up [E*2I, H] and down [E*H, I] "
                         "for the %d experts held", expert_count);
    const int routes = tokens * top_k;
    const int gh = hidden_size / 128, gi = intermediate / 128;
    // small routing state in one block
    const size_t o_logits = 0;
    const size_t o_idx = align_up(o_logits + sizeof(float) * tokens * num_experts, 256);
    const size_t o_w = align_up(o_idx + sizeof(int32_t) * routes, 256);
    const size_t o_off = align_up(o_w + sizeof(float) * routes, 256);
    const size_t o_rt = align_up(o_off + sizeof(int32_t) * (num_experts + 1), 256);
    const size_t o_pos = align_up(o_rt + sizeof(int32_t) * routes, 256);
    const size_t o_act = align_up(o_pos + sizeof(int32_t) * routes, 256);
    const size_t small_bytes = align_up(o_act + sizeof(int4) * num_experts, 256);
    // quantised hidden (per token) and quantised SwiGLU output (per route)
    // The reference's rule (ctx->moe_rule == B2W4_ACT_G32): an expert that holds several routes
    // quantises per 32 values, a lone route per 128; with one token every expert holds one
    // route.  B2W4_ACT_G128: per 128 for every route.
    const bool rule32 = ctx->moe_rule == B2W4_ACT_G32 && tokens >= 2;
    const size_t o_qh = 0;
    const size_t o_ash = align_up(o_qh + (size_t)tokens * hidden_size, 256);
    const size_t o_qi = align_up(o_ash + sizeof(float) * tokens * gh, 256);
    const size_t o_asi = align_up(o_qi + (size_t)routes * intermediate, 256);
    const size_t o_qh32 = align_up(o_asi + sizeof(float) * routes * gi * 4, 256);
    const size_t o_ash32 = align_up(o_qh32 + (rule32 ? (size_t)tokens * hidden_size : 0), 256);
    const size_t quant_bytes =
        align_up(o_ash32 + (rule32 ? sizeof(float) * tokens * gh * 4 : 0), 256);
    void *sm = nullptr, *qb = nullptr, *gu = nullptr, *dn = nullptr;
    int rc;
    if ((rc = b2w4_reserve(ctx, SCR_MOE_A, small_bytes, &sm)) != B2W4_OK ||
        (rc = b2w4_reserve(ctx, SCR_MOE_B, quant_bytes, &qb)) != B2W4_OK ||
        (rc = b2w4_reserve(ctx, SCR_MOE_C, sizeof(float) * (size_t)routes * 2 * intermediate,
                           &gu)) != B2W4_OK ||
        (rc = b2w4_reserve(ctx, SCR_MOE_D, sizeof(float) * (size_t)routes * hidden_size,
                           &dn)) != B2W4_OK)
        return rc;
    uint8_t* smb = static_cast<uint8_t*>(sm);
    uint8_t* qbb = static_cast<uint8_t*>(qb);
    float* logits = reinterpret_cast<float*>(smb + o_logits);
    int32_t* idx = reinterpret_cast<int32_t*>(smb + o_idx);
    float* wts = reinterpret_cast<float*>(smb + o_w);
    int32_t* offsets = reinterpret_cast<int32_t*>(smb + o_off);
    int32_t* route_token = reinterpret_cast<int32_t*>(smb + o_rt);
    int32_t* pos = reinterpret_cast<int32_t*>(smb + o_pos);
    int4* slots = reinterpret_cast<int4*>(smb + o_act);
    int8_t* q_hidden = reinterpret_cast<int8_t*>(qbb + o_qh);
    float* as_hidden = reinterpret_cast<float*>(qbb + o_ash);
    int8_t* q_inter = reinterpret_cast<int8_t*>(qbb + o_qi);
    float* as_inter = reinterpret_cast<float*>(qbb + o_asi);  // [routes][4 * gi]
    int8_t* q_hidden32 = rule32 ? reinterpret_cast<int8_t*>(qbb + o_qh32) : nullptr;
    float* as_hidden32 = rule32 ? reinterpret_cast<float*>(qbb + o_ash32) : nullptr;
    cudaStream_t st = ctx->stream;

    const __half* router = static_cast<const __half*>(router_fp16_dev);
    const bool aligned =
        (reinterpret_cast<uintptr_t>(hidden_dev) | reinterpret_cast<uintptr_t>(router)) % 16 == 0 &&
        ldx % 4 == 0;
    const bool fused = aligned && tokens <= kFusedTokens && routes <= kFusedRoutes;
    // compact positions stay global; the grouped kernels skip experts held elsewhere
    const int32_t* local_offsets = offsets + expert_begin;
    const bool partial = expert_count != num_experts;
    // One token with all experts here: routes need no compaction, each block of the first expert
    // matmul picks its own, and the second one combines its rows.  Measured: 8 of 128 experts of
    // 768, rows of 2048, 22.6 -> 17.8 us for one token again and again (19.9 with a combine launch), a
    // call on its own 27.6 -> 21.5, with experts that no call before had 28.7 -> 23.6, with nothing in
    // L2 29.7 -> 25.7.  In a graph, tokens of other experts in turn, weights not in L2: 22.5 -> 17.3; 8
    // of 64 of 1024, 3072, 30.6 -> 25.4; 8 of 128 of 1536, 4096, 49.1 -> 48.9; 4 of 64 of 384, 1024,
    // 18.5 -> 15.5.  Tried: the second matmul's weights brought to L2 by the first (no gain).
    const bool single = fused && tokens == 1 && !partial && !peers && !route_out;
    const bool in_cluster = single && top_k <= kCombineCluster;
    const TokenRoutes first = {logits, idx, wts, nullptr};
    const TokenRoutes second = {nullptr, idx, wts, in_cluster ? out_dev : nullptr};
    if (fused) {
        // enough blocks to spread the router rows over the SMs, one warp per expert
        const int blocks = (num_experts + kFusedThreads / 32 - 1) / (kFusedThreads / 32);
        B2W4_CUDA(ctx, b2w4_launch_chained(
                           ctx->pdl, single ? moe_route_fused_kernel<false>
                                            : moe_route_fused_kernel<true>,
                           dim3(blocks), dim3(kFusedThreads),
                           sizeof(int) * (num_experts + 1), st, hidden_dev, ldx, tokens,
                           hidden_size, router, num_experts, top_k, logits, idx, wts, offsets,
                           route_token, pos, slots, q_hidden, as_hidden, ctx->flag_dev + 4));
        ctx->launches++;
    } else {
        if (!aligned) {
            const long long threads = (long long)tokens * num_experts * 32;
            B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_router_logits_scalar_kernel,
                                               dim3((int)((threads + 255) / 256)), dim3(256), 0, st,
                                               hidden_dev, ldx, tokens, hidden_size, router,
                                               num_experts, logits));
        } else if (tokens <= 8) {  // decode: one expert per warp keeps every SM busy
            const long long warps = (long long)((tokens + kRouterTok - 1) / kRouterTok) * num_experts;
            B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_router_logits_kernel<1>,
                                               dim3((int)((warps * 32 + 127) / 128)), dim3(128), 0, st,
                                               hidden_dev, ldx, tokens, hidden_size, router,
                                               num_experts, logits));
        } else {
            const long long warps =
                (long long)((tokens + kRouterTok - 1) / kRouterTok) * ((num_experts + 3) / 4);
            B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_router_logits_kernel<4>,
                                               dim3((int)((warps * 32 + 127) / 128)), dim3(128), 0, st,
                                               hidden_dev, ldx, tokens, hidden_size, router,
                                               num_experts, logits));
        }
        ctx->launches++;
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_select_routes_kernel, dim3((tokens + 3) / 4),
                                           dim3(128), 0, st, logits, tokens, num_experts, top_k, idx,
                                           wts));
        ctx->launches++;
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_compact_kernel, dim3(num_experts),
                                           dim3(kCompactThreads), 0, st, idx, tokens, top_k,
                                           num_experts, offsets, route_token, pos, slots));
        ctx->launches++;
    }
    // which grouped-matmul variant: the few-token one implements the per-128 rule only
    const bool decode = rule32 ? false : tokens <= kFusedSwigluTokens;
    // (the fused routing kernel has quantised the rows, per 128 values)
    if (rule32 || !fused) {
        const long long threads = (long long)tokens * gh * 32;
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_quantize_hidden_kernel,
                                           dim3((int)((threads + 255) / 256)), dim3(256), 0, st,
                                           hidden_dev, ldx, tokens, hidden_size, q_hidden,
                                           as_hidden, q_hidden32, as_hidden32));
        ctx->launches++;
    }
    if ((rc = launch_grouped(ctx, gate_up, num_experts, expert_begin, expert_count, routes,
                             q_hidden, as_hidden, gh, q_hidden32, as_hidden32, gh * 4, slots,
                             single ? nullptr : route_token, static_cast<float*>(gu), decode,
                             nullptr, nullptr, 0, single ? &first : nullptr)) != B2W4_OK)
        return rc;
    // few routes: SwiGLU and its quantiser run inside the down-projection's CTAs
    const bool fuse_swiglu = decode;
    if (!fuse_swiglu) {
        const long long threads = (long long)routes * gi * 32;
        B2W4_CUDA(ctx, b2w4_launch_chained(
                           ctx->pdl, moe_swiglu_quant_kernel, dim3((int)((threads + 255) / 256)),
                           dim3(256), 0, st, static_cast<const float*>(gu), routes, intermediate,
                           q_inter, as_inter, gi * 4,
                           rule32 ? static_cast<const int32_t*>(offsets) : nullptr, num_experts,
                           partial ? local_offsets : nullptr,
                           partial ? local_offsets + expert_count : nullptr));
        ctx->launches++;
    }
    // decode steps hand the rows over from the down-projection's own epilogue
    const bool fused_handover = peers != nullptr && decode;
    // a route's SwiGLU row was quantised by its own expert's rule: one code buffer serves both
    if ((rc = launch_grouped(ctx, down, num_experts, expert_begin, expert_count, routes, q_inter,
                             as_inter, gi * 4, rule32 ? q_inter : nullptr,
                             rule32 ? as_inter : nullptr, gi * 4, slots, nullptr,
                             static_cast<float*>(dn), decode,
                             fuse_swiglu ? static_cast<const float*>(gu) : nullptr,
                             fused_handover ? peers : nullptr, stage_rows,
                             single ? &second : nullptr)) != B2W4_OK)
        return rc;
    if (route_out) {
        dim3 grid((hidden_size / 4 + 255) / 256, routes);
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_scatter_routes_kernel, grid, dim3(256), 0,
                                           st, static_cast<const float*>(dn), idx, pos, routes,
                                           hidden_size, expert_begin, expert_count, route_out));
        ctx->launches++;
    }
    if (peers) {
        if (!fused_handover) {
            dim3 sgrid((hidden_size / 4 + 255) / 256, routes);
            B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_scatter_routes_peers_kernel, sgrid,
                                               dim3(256), 0, st, static_cast<const float*>(dn),
                                               idx, pos, routes, hidden_size, expert_begin,
                                               expert_count, stage_rows, *peers));
            ctx->launches++;
        }
        dim3 cgrid((hidden_size / 4 + kCombineThreads - 1) / kCombineThreads, tokens);
        B2W4_CUDA(ctx, b2w4_launch_chained(
                           ctx->pdl, moe_combine_staged_kernel, cgrid, dim3(kCombineThreads), 0, st,
                           peers->stage_peer[peers->rank], stage_rows, idx, wts,
                           fused_handover ? static_cast<const int32_t*>(pos) : nullptr, tokens,
                           top_k, hidden_size, out_dev, ldo,
                           reinterpret_cast<unsigned*>(ctx->flag_dev + 6), ctx->status_dev,
                           ctx->peer_wait_cycles));
        ctx->launches++;
    } else if (out_dev && !in_cluster) {
        dim3 grid((hidden_size / 4 + kCombineThreads - 1) / kCombineThreads, tokens);
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_combine_kernel, grid,
                                           dim3(kCombineThreads), 0, st,
                                           static_cast<const float*>(dn), idx, wts,
                                           single ? nullptr : pos, tokens, top_k, hidden_size,
                                           out_dev, ldo));
        ctx->launches++;
    }
    B2W4_CUDA(ctx, cudaGetLastError());
    if (logits_dev)
        B2W4_CUDA(ctx, cudaMemcpyAsync(logits_dev, logits,
                                       sizeof(float) * (size_t)tokens * num_experts,
                                       cudaMemcpyDeviceToDevice, st));
    if (indices_dev)
        B2W4_CUDA(ctx, cudaMemcpyAsync(indices_dev, idx, sizeof(int32_t) * (size_t)routes,
                                       cudaMemcpyDeviceToDevice, st));
    if (weights_dev)
        B2W4_CUDA(ctx, cudaMemcpyAsync(weights_dev, wts, sizeof(float) * (size_t)routes,
                                       cudaMemcpyDeviceToDevice, st));
    return B2W4_OK;
}

extern "C" {

int b2w4_moe_forward(b2w4_ctx* ctx, const float* hidden_dev, int ldx, int tokens,
                     int hidden_size, const void* router_fp16_dev, int num_experts, int top_k,
                     int intermediate, const b2w4_weight* gate_up, const b2w4_weight* down,
                     float* out_dev, int ldo, float* logits_dev, int32_t* indices_dev,
                     float* weights_dev) {
    if (ctx && !out_dev)
        return b2w4_fail(ctx, B2W4_E_INVALID, "moe: null argument");
    return moe_run(ctx, hidden_dev, ldx, tokens, hidden_size, router_fp16_dev, num_experts,
                   top_k, intermediate, gate_up, down, 0, num_experts, out_dev, ldo, nullptr,
                   logits_dev, indices_dev, weights_dev);
}

int b2w4_moe_expert_outputs(b2w4_ctx* ctx, const float* hidden_dev, int ldx, int tokens,
                            int hidden_size, const void* router_fp16_dev, int num_experts,
                            int top_k, int intermediate, const b2w4_weight* gate_up_local,
                            const b2w4_weight* down_local, int expert_begin, int expert_count,
                            float* route_out_dev, int32_t* indices_dev, float* weights_dev) {
    if (ctx && (!route_out_dev || !indices_dev || !weights_dev))
        return b2w4_fail(ctx, B2W4_E_INVALID, "moe: null argument");
    return moe_run(ctx, hidden_dev, ldx, tokens, hidden_size, router_fp16_dev, num_experts,
                   top_k, intermediate, gate_up_local, down_local, expert_begin, expert_count,
                   nullptr, 0, route_out_dev, nullptr, indices_dev, weights_dev);
}

int b2w4_moe_forward_ep(b2w4_ctx* ctx, const float* hidden_dev, int ldx, int tokens,
                        int hidden_size, const void* router_fp16_dev, int num_experts, int top_k,
                        int intermediate, const b2w4_weight* gate_up_local,
                        const b2w4_weight* down_local, int expert_begin, int expert_count,
                        const b2w4_tp_group* group, int stage_rows, float* out_dev, int ldo,
                        int32_t* indices_dev, float* weights_dev) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!out_dev || !group || group->world < 1 || group->world > kTpMaxWorld ||
        group->rank < 0 || group->rank >= group->world || tokens <= 0 || top_k <= 0 ||
        stage_rows < tokens * top_k)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "moe_forward_ep: bad group, or fewer staging rows than routes");
    b2w4_tp_args peers = {};
    for (int p = 0; p < group->world; ++p) {
        if (!group->stage_peers[p] || (reinterpret_cast<uintptr_t>(group->stage_peers[p]) & 15))
            return b2w4_fail(ctx, B2W4_E_INVALID,
                             "moe_forward_ep: null peer pointer, or not 16-byte aligned");
        peers.stage_peer[p] = static_cast<unsigned long long*>(group->stage_peers[p]);
    }
    peers.world = group->world;
    peers.rank = group->rank;
    return moe_run(ctx, hidden_dev, ldx, tokens, hidden_size, router_fp16_dev, num_experts,
                   top_k, intermediate, gate_up_local, down_local, expert_begin, expert_count,
                   out_dev, ldo, nullptr, nullptr, indices_dev, weights_dev, &peers, stage_rows);
}

int b2w4_moe_combine(b2w4_ctx* ctx, const float* route_out_dev, int tokens, int hidden_size,
                     int top_k, const int32_t* indices_dev, const float* weights_dev,
                     float* out_dev, int ldo) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!route_out_dev || !indices_dev || !weights_dev || !out_dev || tokens <= 0 ||
        hidden_size <= 0 || hidden_size % 4 || top_k <= 0 || top_k > kMaxTopK ||
        ldo < hidden_size || reinterpret_cast<uintptr_t>(route_out_dev) % 16)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "moe_combine: bad argument (hidden a multiple of 4, route rows "
                         "16-byte aligned)");
    dim3 grid((hidden_size / 4 + kCombineThreads - 1) / kCombineThreads, tokens);
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, moe_combine_kernel, grid, dim3(kCombineThreads),
                                       0, ctx->stream, route_out_dev, indices_dev, weights_dev,
                                       static_cast<const int32_t*>(nullptr), tokens, top_k,
                                       hidden_size, out_dev, ldo));
    ctx->launches++;
    B2W4_CUDA(ctx, cudaGetLastError());
    return B2W4_OK;
}

}  // extern "C"
