// The operators that sit between the W4G128 matmuls of a decoder layer, as device kernels, so
// that a decode step needs no trip to the host between its matmuls: RMSNorm, residual add +
// RMSNorm, SwiGLU, add / multiply, rotary embedding, KV-cache append, scaled-dot-product
// attention over the cache, embedding-row lookup.  Semantics follow the reference's CPU
// operators (the x86 build: its scalar and AVX-512 paths), cited per kernel.  Sums over a row
// are tree reductions here where the reference's scalar loops are sequential, so these ops
// agree with the reference to fp32 rounding of a reassociated sum, not bit for bit (attention:
// dot products, and in some forms a softmax over parts of the keys); everything element-wise
// (rotary embedding, add, multiply) uses the reference's operation order with no contraction.
// All tensors are fp32, rows = tokens, features contiguous.
#include "attention_tile.cuh"

#include <cfloat>
#include <type_traits>

#include <cooperative_groups.h>

namespace {

constexpr int kNormThreads = 256;
constexpr int kAttnMaxDim = 256;  // widest attention head

__device__ __forceinline__ float block_sum(float v, float* s_part) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, off));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();  // s_part may still be read from a previous call
    if (lane == 0)
        s_part[warp] = v;
    __syncthreads();
    float t = 0.f;
    const int warps = (blockDim.x + 31) >> 5;
    for (int w = 0; w < warps; ++w)  // every thread adds in the same order
        t = __fadd_rn(t, s_part[w]);
    return t;
}

__device__ __forceinline__ float block_max(float v, float* s_part) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, off));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
    if (lane == 0)
        s_part[warp] = v;
    __syncthreads();
    float t = s_part[0];
    const int warps = (blockDim.x + 31) >> 5;
    for (int w = 1; w < warps; ++w)
        t = fmaxf(t, s_part[w]);
    return t;
}

// kernel_rms_norm (kernels/norm.cpp:13-31, :95-121): r = 1/sqrt(sum(x^2)/D + eps),
// out = (x * r) * w.  With `update`: kernel_add_rms_norm (:123-190): the sum x + update is
// written to `sum` (x itself: the residual stream in place) first.  One block per row.
__global__ void __launch_bounds__(kNormThreads)
rms_norm_kernel(const float* x, int ldx, const float* __restrict__ update, int ldu, float* sum,
                int dim, const float* __restrict__ weight, float eps, float* __restrict__ out,
                int ldo) {
    b2w4_pdl_chain_entry();
    __shared__ float s_part[kNormThreads / 32];
    const float* xr = x + (size_t)blockIdx.x * ldx;
    float* sr = sum + (size_t)blockIdx.x * ldx;
    const float* ur = update ? update + (size_t)blockIdx.x * ldu : nullptr;
    float* orow = out + (size_t)blockIdx.x * ldo;
    // up to kNormHeld values per thread stay in registers between the two passes, all their
    // loads in flight together; longer rows re-read the row
    constexpr int kNormHeld = 16;
    float ss = 0.f;
    if (dim <= kNormHeld * kNormThreads) {
        float v[kNormHeld], w[kNormHeld];
#pragma unroll
        for (int u = 0; u < kNormHeld; ++u) {
            const int d = threadIdx.x + kNormThreads * u;
            v[u] = d < dim ? xr[d] : 0.f;
            w[u] = d < dim ? weight[d] : 0.f;
        }
        if (ur) {
#pragma unroll
            for (int u = 0; u < kNormHeld; ++u) {
                const int d = threadIdx.x + kNormThreads * u;
                if (d < dim) {
                    v[u] = __fadd_rn(v[u], ur[d]);
                    sr[d] = v[u];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kNormHeld; ++u)  // the same per-thread order as the strided loop
            if (threadIdx.x + kNormThreads * u < dim)
                ss = __fadd_rn(ss, __fmul_rn(v[u], v[u]));
        ss = block_sum(ss, s_part);
        const float r = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)dim), eps)));
#pragma unroll
        for (int u = 0; u < kNormHeld; ++u) {
            const int d = threadIdx.x + kNormThreads * u;
            if (d < dim)
                orow[d] = __fmul_rn(__fmul_rn(v[u], r), w[u]);
        }
        return;
    }
    for (int d = threadIdx.x; d < dim; d += blockDim.x) {
        float v = xr[d];
        if (ur) {
            v = __fadd_rn(v, ur[d]);
            sr[d] = v;
        }
        ss = __fadd_rn(ss, __fmul_rn(v, v));
    }
    ss = block_sum(ss, s_part);
    const float r = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)dim), eps)));
    for (int d = threadIdx.x; d < dim; d += blockDim.x)
        orow[d] = __fmul_rn(__fmul_rn(ur ? sr[d] : xr[d], r), weight[d]);
}

// Small rows (the per-head Q/K norm: 128 values): one warp per row.
__global__ void rms_norm_warp_kernel(const float* __restrict__ x, int ldx, int rows, int dim,
                                     const float* __restrict__ weight, float eps,
                                     float* __restrict__ out, int ldo) {
    b2w4_pdl_chain_entry();
    const int row = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= rows)
        return;
    const float* xr = x + (size_t)row * ldx;
    float ss = 0.f;
    for (int d = lane; d < dim; d += 32)
        ss = __fadd_rn(ss, __fmul_rn(xr[d], xr[d]));
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, off));
    const float r = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)dim), eps)));
    float* orow = out + (size_t)row * ldo;
    for (int d = lane; d < dim; d += 32)
        orow[d] = __fmul_rn(__fmul_rn(xr[d], r), weight[d]);
}

// SWIGLU of kernel_elementwise (kernels/elementwise.cpp:529-570): a merged row [2I] holds gate
// = [0, I) and up = [I, 2I); out[i] = (g / (1 + exp(-g))) * up[i] -- a division, unlike the
// MoE op's and the matmul epilogue's g * (1 / (1 + exp(-g))).
__global__ void swiglu_kernel(const float* __restrict__ merged, int ldm, int rows, int inter,
                              float* __restrict__ out, int ldo) {
    b2w4_pdl_chain_entry();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * inter)
        return;
    const int r = (int)(i / inter), c = (int)(i - (size_t)r * inter);
    const float g = merged[(size_t)r * ldm + c];
    const float u = merged[(size_t)r * ldm + inter + c];
    out[(size_t)r * ldo + c] = b2w4_swiglu_value(g, u);
}

__global__ void binary_kernel(const float* __restrict__ a, const float* __restrict__ b,
                              float* __restrict__ out, size_t count, int multiply) {
    b2w4_pdl_chain_entry();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count)
        out[i] = multiply ? __fmul_rn(a[i], b[i]) : __fadd_rn(a[i], b[i]);
}

// kernel_rope, halves form (kernels/rope.cpp:11-50, interleave == false as the Qwen3 graphs
// use it, models/qwen3.py:332-333): out[i] = x0*c - x1*s, out[i+half] = x0*s + x1*c with
// x0 = x[i], x1 = x[i+half]; features beyond rope_dim are copied.  x: [tokens][heads][dim],
// cos / sin: tables [positions][rope_dim/2]; token t uses row pos0 + t, or *pos_dev + t when
// the position lives on the device (a decode step captured once in a CUDA graph and replayed
// for every position).  In place when out == x.
__global__ void rope_kernel(const float* __restrict__ x, float* __restrict__ out, int tokens,
                            int heads, int dim, const float* __restrict__ cosv,
                            const float* __restrict__ sinv, int rope_dim, int pos0,
                            const int* __restrict__ pos_dev) {
    b2w4_pdl_chain_entry();
    const int half = rope_dim >> 1;
    const int pos = pos_dev ? *pos_dev : pos0;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t per_row = (size_t)half + (size_t)(dim - rope_dim);
    if (i >= (size_t)tokens * heads * per_row)
        return;
    const size_t rowi = i / per_row;
    const int j = (int)(i - rowi * per_row);
    const int t = pos + (int)(rowi / heads);
    const float* xr = x + rowi * dim;
    float* orow = out + rowi * dim;
    if (j < half) {
        const float x0 = xr[j], x1 = xr[j + half];
        const float c = cosv[(size_t)t * half + j], s = sinv[(size_t)t * half + j];
        orow[j] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
        orow[j + half] = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
    } else {
        orow[rope_dim + (j - half)] = xr[rope_dim + (j - half)];
    }
}

// KV-cache append: the new tokens' keys and values [tokens][kv_heads][dim] go to positions
// past .. past+tokens-1 of a cache laid out [kv_head][capacity][dim], the layout of the
// reference's cache after its header (kernels/attention.cpp:1043-1057).
__global__ void kv_append_kernel(const float* __restrict__ k, const float* __restrict__ v,
                                 float* __restrict__ k_cache, float* __restrict__ v_cache,
                                 int tokens, int kv_heads, int dim, int past0,
                                 const int* __restrict__ past_dev, int capacity) {
    b2w4_pdl_chain_entry();
    const int past = past_dev ? min(*past_dev, capacity - tokens) : past0;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)tokens * kv_heads * dim)
        return;
    const int d = (int)(i % dim);
    const int h = (int)((i / dim) % kv_heads);
    const int t = (int)(i / ((size_t)dim * kv_heads));
    const size_t dst = ((size_t)h * capacity + past + t) * dim + d;
    k_cache[dst] = k[i];
    v_cache[dst] = v[i];
}

// The step between the fused qkv matmul and attention in one launch (the reference's CUDA
// backend fuses Q/K norm and rotary embedding the same way, engine/cuda_attention.cu:8-55):
// per (token, head) row of the merged qkv output -- a warp each -- the Q and K rows get the
// per-head RMSNorm (weights optional) and the rotary embedding, with exactly the operations of
// rms_norm_warp_kernel and rope_kernel in their order, Q goes to q_out [tokens][heads][dim],
// K and V go straight to their cache rows.  Needs rope over the whole head and dim / 2 a
// multiple of 32, so that both halves of a rotary pair sit in one lane.  The head size is a
// constant of the kernel and indices have 32 bits: 1500 tokens of 32 / 8 heads of 128 took 28 us
// with a size read at run time and 64-bit divisions.
// One query or key row, by one warp; stored to dst.
template <int DIM>
__device__ __forceinline__ void prepare_row(const float* __restrict__ x,
                                            const float* __restrict__ w, float eps,
                                            const float* __restrict__ cosv,
                                            const float* __restrict__ sinv, int lane,
                                            float* __restrict__ dst) {
    constexpr int kPer = DIM / 32, kHi = kPer / 2;  // v[i] pairs with v[i + kHi]
    float v[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i)
        v[i] = x[lane + 32 * i];
    if (w) {
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < kPer; ++i)
            ss = __fadd_rn(ss, __fmul_rn(v[i], v[i]));
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, off));
        const float r = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)DIM), eps)));
#pragma unroll
        for (int i = 0; i < kPer; ++i)
            v[i] = __fmul_rn(__fmul_rn(v[i], r), w[lane + 32 * i]);
    }
#pragma unroll
    for (int i = 0; i < kHi; ++i) {
        const int j = lane + 32 * i;
        const float c = cosv[j], sn = sinv[j];
        dst[j] = __fsub_rn(__fmul_rn(v[i], c), __fmul_rn(v[i + kHi], sn));
        dst[j + DIM / 2] = __fadd_rn(__fmul_rn(v[i], sn), __fmul_rn(v[i + kHi], c));
    }
}

template <int DIM>
__global__ void __launch_bounds__(256)
qkv_prepare_kernel(const float* __restrict__ qkv, int ld, unsigned tokens, int heads, int kv_heads,
                   const float* __restrict__ q_weight, const float* __restrict__ k_weight,
                   float eps, const float* __restrict__ cosv, const float* __restrict__ sinv,
                   int pos0, const int* __restrict__ pos_dev, float* __restrict__ q_out,
                   float* __restrict__ k_cache, float* __restrict__ v_cache, int capacity) {
    b2w4_pdl_chain_entry();
    const unsigned slots = heads + 2 * kv_heads;
    const unsigned row = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= tokens * slots)
        return;
    const int pos = pos_dev ? min(*pos_dev, capacity - (int)tokens) : pos0;
    const int t = (int)(row / slots), slot = (int)(row - t * slots);
    const float* x = qkv + (size_t)t * ld + (size_t)slot * DIM;
    if (slot >= heads + kv_heads) {  // a value row: copied to its cache row
        float* dst = v_cache + ((size_t)(slot - heads - kv_heads) * capacity + pos + t) * DIM;
#pragma unroll
        for (int i = 0; i < DIM; i += 32)
            dst[lane + i] = x[lane + i];
        return;
    }
    const bool is_q = slot < heads;
    prepare_row<DIM>(x, is_q ? q_weight : k_weight, eps, cosv + (size_t)(pos + t) * (DIM / 2),
                     sinv + (size_t)(pos + t) * (DIM / 2), lane,
                     is_q ? q_out + ((size_t)t * heads + slot) * DIM
                          : k_cache + ((size_t)(slot - heads) * capacity + pos + t) * DIM);
}

// Scaled-dot-product attention of one (query token, head) over the cache, the x86 reference's
// arithmetic (kernels/attention_x86_avx512.cpp:47-109): scores = dot(q, k_j) * scale for the
// visible keys (causal: keys 0 .. past + t), full-row softmax (max, exp, sum, times 1/sum),
// then out = sum_j p_j * v_j accumulated key by key in ascending order with one fused
// multiply-add per key and feature, as the reference's loop does; a probability of zero
// contributes nothing.  One block per (token, head): the form that takes any head size and
// any alignment.  Scores: a warp per key, four keys' loads in flight at a time.  P*V: thread d
// owns output feature d and walks the keys in order; the value rows come through shared memory
// in chunks that all threads fetch together, the next chunk's loads in flight while the current
// one is consumed, so that the ordered sum does not wait on memory once per key.
// What bounds it: the latency of those loads (16 KB in flight per block).  Keys staged through
// shared memory with a lane per 32 features and a running softmax, so that the sums follow
// attention_tile_kernel's order, was slower on every shape that takes this form: 32 / 8 heads
// of 80, one token behind 1000 keys 71 us against 42, 32 tokens 318 against 140; of 96 tokens
// behind 6000 keys 2028 against 830.
constexpr int kAttnWarps = kAttnThreads / 32;
constexpr int kAttnStage = 4096;                       // floats of V per chunk
constexpr int kAttnPerThread = kAttnStage / kAttnThreads;
__global__ void __launch_bounds__(kAttnThreads)
attention_kernel(const float* __restrict__ q, const float* __restrict__ k_cache,
                 const float* __restrict__ v_cache, float* __restrict__ out, int tokens,
                 int heads, int kv_heads, int dim, int past0, const int* __restrict__ past_dev,
                 int capacity, float scale, int score_slots) {
    b2w4_pdl_chain_entry();
    const int past = past_dev ? min(*past_dev, capacity - tokens) : past0;
    extern __shared__ float s_dyn[];
    float* s_scores = s_dyn;                // [score_slots] >= visible keys
    float* s_stage = s_dyn + score_slots;   // [kAttnStage]
    __shared__ float s_part[kAttnWarps];
    const int t = blockIdx.x / heads, h = blockIdx.x % heads;
    const int kvh = h / (heads / kv_heads);
    const int visible = past + t + 1;
    const float* qr = q + ((size_t)t * heads + h) * dim;
    const float* kc = k_cache + (size_t)kvh * capacity * dim;
    const float* vc = v_cache + (size_t)kvh * capacity * dim;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    constexpr int kQ = kAttnMaxDim / 32, kKeys = 4;
    float qv[kQ];
#pragma unroll
    for (int i = 0; i < kQ; ++i)
        qv[i] = lane + 32 * i < dim ? qr[lane + 32 * i] : 0.f;
    for (int j0 = warp * kKeys; j0 < visible; j0 += kAttnWarps * kKeys) {
        float kv[kKeys][kQ];
#pragma unroll
        for (int u = 0; u < kKeys; ++u)
#pragma unroll
            for (int i = 0; i < kQ; ++i)
                kv[u][i] = (j0 + u < visible && lane + 32 * i < dim)
                               ? kc[(size_t)(j0 + u) * dim + lane + 32 * i] : 0.f;
#pragma unroll
        for (int u = 0; u < kKeys; ++u) {
            float p = 0.f;
#pragma unroll
            for (int i = 0; i < kQ; ++i)
                if (32 * i < dim)  // lanes past the last feature add +0 products
                    p = __fmaf_rn(qv[i], kv[u][i], p);
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                p = __fadd_rn(p, __shfl_xor_sync(0xffffffffu, p, off));
            if (lane == 0 && j0 + u < visible)
                s_scores[j0 + u] = __fmul_rn(p, scale);
        }
    }
    __syncthreads();
    float m = -INFINITY;
    for (int j = threadIdx.x; j < visible; j += blockDim.x)
        m = fmaxf(m, s_scores[j]);
    m = block_max(m, s_part);
    float sum = 0.f;
    for (int j = threadIdx.x; j < visible; j += blockDim.x) {
        const float e = (float)exp((double)__fsub_rn(s_scores[j], m));
        s_scores[j] = e;
        sum = __fadd_rn(sum, e);
    }
    sum = block_sum(sum, s_part);
    const float inv = __fdiv_rn(1.f, sum);

    const int chunk = kAttnStage / dim;  // keys per chunk
    float r[kAttnPerThread];
    auto fetch = [&](int j0) {
        const int n = min(chunk, visible - j0) * dim;
        const float* src = vc + (size_t)j0 * dim;
#pragma unroll
        for (int u = 0; u < kAttnPerThread; ++u) {
            const int i = threadIdx.x + kAttnThreads * u;
            r[u] = i < n ? src[i] : 0.f;
        }
    };
    fetch(0);
    float acc = 0.f;
    for (int j0 = 0; j0 < visible; j0 += chunk) {
        __syncthreads();  // the previous chunk has been consumed (and the scores are final)
#pragma unroll
        for (int u = 0; u < kAttnPerThread; ++u)
            s_stage[threadIdx.x + kAttnThreads * u] = r[u];
        __syncthreads();
        if (j0 + chunk < visible)
            fetch(j0 + chunk);
        if (threadIdx.x < dim) {
            const int nk = min(chunk, visible - j0);
            for (int j = 0; j < nk; ++j) {
                const float p = __fmul_rn(s_scores[j0 + j], inv);
                if (p != 0.f)
                    acc = __fmaf_rn(s_stage[j * dim + threadIdx.x], p, acc);
            }
        }
    }
    if (threadIdx.x < dim)
        out[((size_t)t * heads + h) * dim + threadIdx.x] = acc;
}

// attention_tile_kernel's arithmetic, operation for operation, one block per (token, head): a
// dot product is summed per 32 features (even and odd ones apart), the parts in order; the
// softmax runs over blocks of keys; a block's probabilities add up in an xor-tree; one division
// at the end.  Written plainly (a thread per key, one warp for the softmax, a thread per
// feature): B2W4_ATTN=row runs it on the head sizes of the tile and cluster kernels, to compare
// them with.
__global__ void __launch_bounds__(kAttnThreads)
attention_plain_kernel(const float* __restrict__ q, const float* __restrict__ k_cache,
                       const float* __restrict__ v_cache, float* __restrict__ out, int tokens,
                       int heads, int kv_heads, int dim, int past0,
                       const int* __restrict__ past_dev, int capacity, float scale,
                       int score_slots) {
    b2w4_pdl_chain_entry();
    const int past = past_dev ? min(*past_dev, capacity - tokens) : past0;
    extern __shared__ float s_dyn[];
    float* s_scores = s_dyn;               // [score_slots] >= visible keys
    float* s_alpha = s_dyn + score_slots;  // [blocks]: factor before block b
    __shared__ float s_max, s_total;
    const int t = blockIdx.x / heads, h = blockIdx.x % heads;
    const int kvh = h / (heads / kv_heads);
    const int visible = past + t + 1, blocks = (visible + kTileKeys - 1) / kTileKeys;
    const float* qr = q + ((size_t)t * heads + h) * dim;
    const float* kc = k_cache + (size_t)kvh * capacity * dim;
    const float* vc = v_cache + (size_t)kvh * capacity * dim;
    const int lane = threadIdx.x & 31;
    auto scores = [&]() {
        for (int j = threadIdx.x; j < visible; j += kAttnThreads) {
            const float* kr = kc + (size_t)j * dim;
            float s = 0.f;
            for (int c = 0; c < dim; c += 32) {
                float even = 0.f, odd = 0.f;
                for (int i = c; i < c + 32; i += 2) {
                    even = __fmaf_rn(qr[i], kr[i], even);
                    odd = __fmaf_rn(qr[i + 1], kr[i + 1], odd);
                }
                s = __fadd_rn(s, __fadd_rn(even, odd));
            }
            s_scores[j] = __fmul_rn(s, scale);
        }
        __syncthreads();
    };
    scores();
    if (threadIdx.x < 32) {
        float m = -INFINITY, l = 0.f;
        for (int b = 0; b < blocks; ++b) {
            const int j = b * kTileKeys + lane;
            float mb = j < visible ? fmaxf(m, s_scores[j]) : m;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1)
                mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, off));
            const float alpha = b ? attn_rescale(m, mb) : 1.f;
            m = mb;
            float e = 0.f;
            if (j < visible)
                s_scores[j] = e = attn_prob(s_scores[j], m);
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
                e = __fadd_rn(e, __shfl_xor_sync(0xffffffffu, e, off));
            l = __fadd_rn(__fmul_rn(l, alpha), e);
            if (lane == 0)
                s_alpha[b] = alpha;
        }
        if (lane == 0) {
            s_max = m;
            s_total = l;
        }
    }
    __syncthreads();
    auto weigh = [&](bool final_pass) {  // thread d: feature d
        float acc = 0.f;
        for (int j = 0; threadIdx.x < dim && j < visible; ++j) {
            if (j % kTileKeys == 0 && !final_pass) {
                const float al = s_alpha[j / kTileKeys];
                acc = al == 0.f ? 0.f : __fmul_rn(acc, al);
            }
            const float p = s_scores[j];
            if (p != 0.f)
                acc = __fmaf_rn(vc[(size_t)j * dim + threadIdx.x], p, acc);
        }
        return final_pass ? acc : __fdiv_rn(acc, s_total);
    };
    float o = weigh(false);
    if (__syncthreads_or(threadIdx.x < dim && !(fabsf(o) <= FLT_MAX))) {
        scores();
        const float inv = __fdiv_rn(1.f, s_total);
        for (int j = threadIdx.x; j < visible; j += kAttnThreads)
            s_scores[j] = __fmul_rn(attn_prob(s_scores[j], s_max), inv);
        __syncthreads();
        o = weigh(true);
    }
    if (threadIdx.x < dim)
        out[((size_t)t * heads + h) * dim + threadIdx.x] = o;
}

// The same attention for few query tokens (a decode step, a short run): one block per (token,
// kv head, up to HR of its query heads), or a cluster of `ctas` blocks that splits the visible
// keys, so that a step fills the chip.  The query heads of a kv head read its keys and values
// once.  What bounds it: bytes in flight -- a key and value row are read once and used HR times
// -- until the cache is short, where it is the chain load, exchange, exp, load, exchange.
//   scores   eight lanes per key hold four features each of every 32, a warp has 4 (KI)
//            x 4 keys' loads in flight; products in pairs (fma.rn.f32x2), then a butterfly
//            over the eight lanes that halves the items held at each level
//   softmax  over the block's own keys: max m, e_j = exp(s_j - m), l = sum e_j
//   P*V      a warp per key, four features per lane, HR accumulator rows; the warps' sums are
//            added through shared memory; the first value rows are fetched before the softmax
//            (6000 keys 22.7 -> 21.4 us)
//   merge    block r adds its share of the features over the cluster (distributed shared
//            memory): out = sum_c w_c o_c / sum_c w_c l_c, w_c = exp(m_c - max m)
// Up to `one_range` visible keys the first block takes them all and the others leave: a cluster
// costs more than it gives there (a step at position 0, 32 / 8 heads of 128: 3.1 us with one
// block per head, 6.2 split over sixteen, 3.0 as it is; seven tokens 3.8, 23.4, 3.3).
// Measured, a step with 32 / 8 heads of 128 behind 6000 keys: 313 us with one block per head
// (32 of 148 SMs, every key read four times), 21.4 us over sixteen blocks, 32 over eight.
// The split depends on the number of visible keys and the call's sizes, so a position given by
// the host and one read on the device leave the same bits.  A probability of zero contributes
// nothing (whatever the value row holds), as in attention_kernel: where a block's sums are not
// finite -- a value row that is not, or values near the largest number added up before the
// division -- every block forms them again from the final probabilities.  A NaN score reaches every
// feature.
// PREP (one token): the rows come straight from the fused qkv matmul.  Every block makes the
// query rows it needs (qkv_prepare_kernel's norm and rotary embedding, a warp per row); the
// block whose keys end with the new one makes that key and value row too and writes them to the
// cache before it reads its keys.  A launch of its own for that costs 2.5 to 3 us a layer.
struct PrepArgs {
    const float *qkv, *q_weight, *k_weight, *cosv, *sinv;
    float eps;
    float *k_cache, *v_cache;
};
// RING: there are no more blocks than multiprocessors, one or two to each, so key and value rows go
// through a ring of slots per warp in their shared memory (cp.async): first the warp's keys, then its
// values, a slot as soon as it has been read, from before the query rows are made to the last value
// row.  No warp waits for another.  The same bits as without: a key's dot product has one order in
// whichever warp it is made (a warp has four keys in a row at 128 features, eight at 64; without the
// ring up to sixteen), and every value stays with its warp and lanes.  What it mends: with loads into registers (8 KB of keys or 4 KB of values in flight per
// warp) each pass over the block's keys waits for its memory round trip, and nothing is on its way
// while the query rows are made.  (By bulk copies, 2 KB of keys or 512 bytes of values each, a step
// of eight layers behind 6000 keys took 581 us instead of 455.)
constexpr int kRingSlots = 5, kSlotBytes = 2048;
constexpr int kMaxRanges = 16;
// blocks per multiprocessor that the registers allow
constexpr int split_blocks(int dim, int hr) { return dim * hr <= 128 ? 4 : dim * hr <= 256 ? 3 : 2; }
template <int DIM, int HR>
struct SplitSmem {  // floats of dynamic shared memory before the scores
    static constexpr int kAcc = 0;                              // [kAttnWarps][HR][DIM]
    static constexpr int kOut = kAcc + kAttnWarps * HR * DIM;   // [HR][DIM]
    static constexpr int kMax = kOut + HR * DIM;                // [HR] m, read by the cluster
    static constexpr int kSum = kMax + HR;                      // [HR] l
    static constexpr int kPart = kSum + HR;                     // [2][kAttnWarps][HR]
    static constexpr int kWeight = kPart + 2 * kAttnWarps * HR;  // [HR][kMaxRanges]
    static constexpr int kTotal = kWeight + HR * kMaxRanges;    // [HR] sum over the cluster
    static constexpr int kOdd = kTotal + HR;                    // 1: not finite; [1]: any block's
    static constexpr int kScores = (kOdd + 2 + 3) & ~3;         // [keys][HR]
};
// k_cache, v_cache: no __restrict__, with PREP the block reads a row that it wrote
template <int DIM, int HR, int CTAS, bool PREP, bool RING>
__global__ void __launch_bounds__(kAttnThreads, RING ? 2 : split_blocks(DIM, HR))
attention_split_kernel(const float* __restrict__ q, const float* k_cache, const float* v_cache,
                       float* __restrict__ out, int tokens, int heads, int kv_heads, int past0,
                       const int* __restrict__ past_dev, int capacity, float scale, int one_range,
                       const PrepArgs prep) {
    b2w4_pdl_chain_entry();
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    const int past = past_dev ? min(*past_dev, capacity - tokens) : past0;
    using S = SplitSmem<DIM, HR>;
    extern __shared__ __align__(16) float s_dyn[];
    float* s_acc = s_dyn + S::kAcc;
    float* s_out = s_dyn + S::kOut;
    float* s_max = s_dyn + S::kMax;
    float* s_sum = s_dyn + S::kSum;
    float* s_part = s_dyn + S::kPart;
    float* s_weight = s_dyn + S::kWeight;
    float* s_total = s_dyn + S::kTotal;
    float* s_odd = s_dyn + S::kOdd;
    float* s_sc = s_dyn + S::kScores;
    const int rep = heads / kv_heads, sets = (rep + HR - 1) / HR;
    const int kvh = blockIdx.y / sets, r0 = (blockIdx.y % sets) * HR;  // heads r0.. of the kv head
    const int nh = min(HR, rep - r0), t = blockIdx.z, rank = blockIdx.x;
    const int visible = past + t + 1;
    const int ranges = CTAS == 1 || visible <= one_range ? 1 : CTAS;
    if (CTAS > 1 && rank >= ranges)  // nobody waits for a block that has left
        return;
    const int per = ranges == 1 ? visible : (visible + CTAS - 1) / CTAS;
    const int j0 = min(rank * per, visible), n = min(per, visible - j0);
    const size_t row0 = ((size_t)t * heads + (size_t)kvh * rep + r0) * DIM;
    const float* kc = k_cache + ((size_t)kvh * capacity + j0) * DIM;
    const float* vc = v_cache + ((size_t)kvh * capacity + j0) * DIM;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    // value rows: a warp per key (two for 64 features)
    constexpr int kLanes = DIM / 4 < 32 ? DIM / 4 : 32;  // lanes per value row
    constexpr int kV4 = DIM / 4 / kLanes;                // float4 per lane
    constexpr int kKeys = 32 / kLanes;                   // keys per warp and step
    // RING: a slot holds kSlotKeys keys in a row, or four value steps, of 512 bytes each
    constexpr int kSlotKeys = kSlotBytes / (DIM * 4), kSlotSteps = kSlotBytes / 512;
    uint8_t* ring = nullptr;
    int key_slots = 0, slots = 0, issued = 0;
    // Copies of slot `i` of the warp's sequence, one group even where there is nothing.
    auto issue = [&](int i) {
        uint8_t* dst = ring + i % kRingSlots * kSlotBytes + lane * 16;
        if (i < slots) {
            const bool keys = i < key_slots;
            const int key0 = (i * kAttnWarps + warp) * kSlotKeys;
            const int step0 = (i - key_slots) * kSlotSteps;
#pragma unroll
            for (int u = 0; u < kSlotSteps; ++u) {  // 512 bytes a step
                const int key = (keys ? key0 + u * kKeys : ((step0 + u) * kAttnWarps + warp) * kKeys) +
                                lane / kLanes;
                if (key < n)
                    cp_async16(reinterpret_cast<float*>(dst + u * 512),
                               (keys ? kc : vc) + (size_t)key * DIM + lane % kLanes * 4, true);
            }
        }
        cp_async_commit();
    };
    const bool owner = n > 0 && j0 + n == visible;  // of the new key, the last one
    if constexpr (RING) {
        ring = reinterpret_cast<uint8_t*>(
                   (reinterpret_cast<uintptr_t>(s_sc + n * HR) + 127) & ~uintptr_t(127)) +
               warp * kRingSlots * kSlotBytes;
        // slots that begin before key n, of every eighth
        auto share = [&](int unit) { return ((n + unit - 1) / unit - warp + kAttnWarps - 1) / kAttnWarps; };
        key_slots = share(kSlotKeys);
        slots = key_slots + (share(kKeys) + kSlotSteps - 1) / kSlotSteps;
        // what does not wait for the new key's row: the keys before its slot
        const bool last = owner && PREP && (n - 1) / kSlotKeys % kAttnWarps == warp;
        issued = min(kRingSlots, !owner || !PREP ? slots : last ? key_slots - 1 : key_slots);
        for (int i = 0; i < issued; ++i)
            issue(i);
    }
    if (PREP) {  // query rows to the head of s_acc, which is free until P*V
        const float* cosv = prep.cosv + (size_t)past * (DIM / 2);
        const float* sinv = prep.sinv + (size_t)past * (DIM / 2);
        const size_t row = ((size_t)kvh * capacity + past) * DIM;
        if (warp < nh) {
            prepare_row<DIM>(prep.qkv + row0 + warp * DIM, prep.q_weight, prep.eps, cosv, sinv,
                             lane, s_acc + warp * DIM);
        } else if (warp == HR && owner) {
            prepare_row<DIM>(prep.qkv + (size_t)(heads + kvh) * DIM, prep.k_weight, prep.eps,
                             cosv, sinv, lane, prep.k_cache + row);
        } else if (warp == HR + 1 && owner) {
            const float* x = prep.qkv + (size_t)(heads + kv_heads + kvh) * DIM;
#pragma unroll
            for (int i = lane; i < DIM; i += 32)
                prep.v_cache[row + i] = x[i];
        }
        __syncthreads();
    }
    if constexpr (RING)
        for (int i = issued; i < kRingSlots; ++i)
            issue(i);
    // Slot i of the warp's sequence, when it is there; after it has been read.
    auto take = [&](int i) {
        cp_async_wait<kRingSlots - 1>();
        __syncwarp();
        return ring + i % kRingSlots * kSlotBytes;
    };
    auto release = [&](int i) {
        __syncwarp();
        issue(i + kRingSlots);
    };

    // ---- scores ----
    {
        constexpr int kF4 = DIM / 32;             // float4 of a row per lane
        const int part = lane & 7, sub = lane >> 3;
        uint64_t qv[HR][2 * kF4];
#pragma unroll
        for (int h = 0; h < HR; ++h)
#pragma unroll
            for (int i = 0; i < kF4; ++i) {
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (h < nh)
                    x = *reinterpret_cast<const float4*>((PREP ? s_acc : q + row0) + h * DIM +
                                                         32 * i + 4 * part);
                qv[h][2 * i] = b2w4_pack2(x.x, x.y);
                qv[h][2 * i + 1] = b2w4_pack2(x.z, x.w);
            }
        // keys per lane group in flight; few keys: one, so that all warps take part
        auto score = [&](auto in_flight) {
            constexpr int KI = decltype(in_flight)::value;
            constexpr int kItems = KI * HR;
            for (int j = warp * 4 * KI, slot = 0; j < n; j += kAttnWarps * 4 * KI, ++slot) {
                float4 kr[KI][kF4];
                // past the end: dropped below
                const float* rows =
                    RING ? reinterpret_cast<const float*>(take(slot)) : kc + (size_t)j * DIM;
#pragma unroll
                for (int it = 0; it < KI; ++it)
#pragma unroll
                    for (int i = 0; i < kF4; ++i) {
                        const int key = RING ? it * 4 + sub : min(it * 4 + sub, n - 1 - j);
                        kr[it][i] = *reinterpret_cast<const float4*>(rows + key * DIM + 32 * i +
                                                                     4 * part);
                    }
                if constexpr (RING)
                    release(slot);
                float v[kItems];  // item it * HR + h
#pragma unroll
                for (int it = 0; it < KI; ++it)
#pragma unroll
                    for (int h = 0; h < HR; ++h) {
                        uint64_t a = 0, b = 0;  // (0.f, 0.f)
#pragma unroll
                        for (int i = 0; i < kF4; ++i) {
                            a = b2w4_fma2(qv[h][2 * i], b2w4_pack2(kr[it][i].x, kr[it][i].y), a);
                            b = b2w4_fma2(qv[h][2 * i + 1], b2w4_pack2(kr[it][i].z, kr[it][i].w), b);
                        }
                        float a0, a1, b0, b1;
                        b2w4_unpack2(a, a0, a1);
                        b2w4_unpack2(b, b0, b1);
                        v[it * HR + h] = __fadd_rn(__fadd_rn(a0, b0), __fadd_rn(a1, b1));
                    }
                int first = 0;  // the lane's first item
                constexpr int kLevel[3] = {4, 2, 1};
#pragma unroll
                for (int l = 0; l < 3; ++l) {
                    const int off = kLevel[l], have = kItems >> l;
                    if (have > 1) {
                        const bool up = lane & off;
#pragma unroll
                        for (int i = 0; i < have / 2; ++i) {
                            const float send = up ? v[i] : v[i + have / 2];
                            const float keep = up ? v[i + have / 2] : v[i];
                            v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, off));
                        }
                        first += up ? have / 2 : 0;
                    } else {
                        v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
                    }
                }
#pragma unroll
                for (int i = 0; i < (kItems > 8 ? kItems / 8 : 1); ++i) {
                    const int item = first + i, key = j + (item / HR) * 4 + sub;
                    if (key < n)
                        s_sc[key * HR + item % HR] = __fmul_rn(v[i], scale);
                }
            }
        };
        if constexpr (RING)
            score(std::integral_constant<int, kSlotKeys / 4>());
        else if (n <= 4 * kAttnWarps)
            score(std::integral_constant<int, 1>());
        else
            score(std::integral_constant<int, (DIM > 128 ? 2 : 4)>());
    }
    __syncthreads();

    // U steps of value rows in flight; the first ones are on their way during the softmax
    constexpr int U = RING ? kSlotSteps : 8 / kV4;
    const int v_part = lane % kLanes, v_sub = lane / kLanes, v_first = warp * kKeys + v_sub;
    float4 vr[U][kV4];
    auto fetch_values = [&](int j) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < kV4; ++i) {
                const int key = min(j + u * kAttnWarps * kKeys, n - 1);
                vr[u][i] = *reinterpret_cast<const float4*>(vc + (size_t)key * DIM +
                                                            4 * (v_part + kLanes * i));
            }
    };
    if (!RING && v_first < n)
        fetch_values(v_first);

    // ---- softmax over the block's keys; a thread's items all belong to head tid % HR ----
    const int my_head = threadIdx.x % HR;
    auto head_reduce = [&](float x, bool maximum) {
#pragma unroll
        for (int off = 16; off >= HR; off >>= 1) {
            const float y = __shfl_xor_sync(0xffffffffu, x, off);
            x = maximum ? fmaxf(x, y) : __fadd_rn(x, y);
        }
        float* parts = s_part + (maximum ? 0 : kAttnWarps * HR);
        if (lane < HR)
            parts[warp * HR + lane] = x;
        __syncthreads();
        x = parts[my_head];
#pragma unroll
        for (int w = 1; w < kAttnWarps; ++w)
            x = maximum ? fmaxf(x, parts[w * HR + my_head])
                        : __fadd_rn(x, parts[w * HR + my_head]);
        return x;
    };
    float m = -INFINITY;
    for (int i = threadIdx.x; i < n * HR; i += kAttnThreads)
        m = fmaxf(m, s_sc[i]);
    m = head_reduce(m, true);
    // scores of -inf only (or none): e_j = exp(-inf) = 0 here, and w_c = 0 unless every
    // block's are, which gives the NaN that attention_kernel gives
    const float base = m == -INFINITY ? 0.f : m;
    float sum = 0.f;
    for (int i = threadIdx.x; i < n * HR; i += kAttnThreads) {
        const float e = (float)exp((double)__fsub_rn(s_sc[i], base));
        s_sc[i] = e;
        sum = __fadd_rn(sum, e);
    }
    sum = head_reduce(sum, false);
    if (threadIdx.x < HR) {
        s_max[threadIdx.x] = m;
        s_sum[threadIdx.x] = sum;
    }
    if (threadIdx.x == 0)
        s_odd[0] = 0.f;

    // ---- P*V ----
    {
        uint64_t acc[HR][2 * kV4];
#pragma unroll
        for (int h = 0; h < HR; ++h)
#pragma unroll
            for (int i = 0; i < 2 * kV4; ++i)
                acc[h][i] = 0;
        for (int j = v_first, slot = key_slots; RING ? slot < slots : j < n;
             j += kAttnWarps * kKeys * U, ++slot) {
            if constexpr (RING) {
                const uint8_t* rows = take(slot);
#pragma unroll
                for (int u = 0; u < U; ++u)
                    vr[u][0] = *reinterpret_cast<const float4*>(rows + u * 512 + lane * 16);
                release(slot);
            } else if (j != v_first) {
                fetch_values(j);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int key = j + u * kAttnWarps * kKeys;
                if (key < n) {
#pragma unroll
                    for (int h = 0; h < HR; ++h) {
                        const float p = s_sc[key * HR + h];
                        if (p != 0.f) {
                            const uint64_t pp = b2w4_pack2(p, p);
#pragma unroll
                            for (int i = 0; i < kV4; ++i) {
                                acc[h][2 * i] = b2w4_fma2(b2w4_pack2(vr[u][i].x, vr[u][i].y), pp,
                                                          acc[h][2 * i]);
                                acc[h][2 * i + 1] =
                                    b2w4_fma2(b2w4_pack2(vr[u][i].z, vr[u][i].w), pp,
                                              acc[h][2 * i + 1]);
                            }
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int h = 0; h < HR; ++h)
#pragma unroll
            for (int i = 0; i < kV4; ++i) {
                float4 o;
                b2w4_unpack2(acc[h][2 * i], o.x, o.y);
                b2w4_unpack2(acc[h][2 * i + 1], o.z, o.w);
                if (kKeys > 1) {  // two keys per step: the half-warps' sums
                    o.x = __fadd_rn(o.x, __shfl_xor_sync(0xffffffffu, o.x, 16));
                    o.y = __fadd_rn(o.y, __shfl_xor_sync(0xffffffffu, o.y, 16));
                    o.z = __fadd_rn(o.z, __shfl_xor_sync(0xffffffffu, o.z, 16));
                    o.w = __fadd_rn(o.w, __shfl_xor_sync(0xffffffffu, o.w, 16));
                }
                if (v_sub == 0)
                    *reinterpret_cast<float4*>(s_acc + (warp * HR + h) * DIM +
                                               4 * (v_part + kLanes * i)) = o;
            }
    }
    __syncthreads();
    // where sums are not finite: once more on final probabilities, zero ones skipped
    auto weigh_again = [&](float* sums) {
#pragma unroll 1
        for (int i = threadIdx.x; i < HR * DIM; i += kAttnThreads) {
            const int h = i / DIM, d = i % DIM;
            float a = 0.f;
#pragma unroll 1
            for (int j = 0; j < n; ++j) {
                const float p = s_sc[j * HR + h];
                if (p != 0.f)
                    a = __fmaf_rn(vc[(size_t)j * DIM + d], p, a);
            }
            sums[i] = a;
        }
    };
    bool odd = false;
    for (int i = threadIdx.x; i < HR * DIM; i += kAttnThreads) {
        float a = s_acc[i];
#pragma unroll
        for (int w = 1; w < kAttnWarps; ++w)
            a = __fadd_rn(a, s_acc[w * HR * DIM + i]);
        if (ranges == 1) {
            a = __fdiv_rn(a, s_sum[i / DIM]);
            if (i / DIM < nh)
                out[row0 + i] = a;
        } else {
            s_out[i] = a;
        }
        odd |= !(fabsf(a) <= FLT_MAX);
    }
    if (ranges == 1) {
        if (__syncthreads_or(odd)) {
            const float inv = __fdiv_rn(1.f, s_sum[my_head]);
            for (int i = threadIdx.x; i < n * HR; i += kAttnThreads)
                s_sc[i] = __fmul_rn(s_sc[i], inv);
            __syncthreads();
            weigh_again(s_out);  // a thread's own sums
            for (int i = threadIdx.x; i < nh * DIM; i += kAttnThreads)
                out[row0 + i] = s_out[i];
        }
        return;
    }
    if (odd)
        s_odd[0] = 1.f;
    cluster.sync();

    // ---- merge ----
    // weights: warp h, head h's; lane c, block c of the cluster
    if (warp < HR) {
        const int c = lane % CTAS;
        const bool in = lane < CTAS;
        const float mc = in ? cluster.map_shared_rank(s_max, c)[warp] : -INFINITY;
        const float lc = in ? cluster.map_shared_rank(s_sum, c)[warp] : 0.f;
        const float any = in ? cluster.map_shared_rank(s_odd, c)[0] : 0.f;
        float top = mc;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
        const float w = (float)exp((double)__fsub_rn(mc, top));
        float l = in ? __fmul_rn(w, lc) : 0.f;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            l = __fadd_rn(l, __shfl_xor_sync(0xffffffffu, l, off));
        if (in)
            s_weight[warp * kMaxRanges + lane] = w;
        if (lane == 0)
            s_total[warp] = l;
        const bool again = __any_sync(0xffffffffu, any != 0.f);
        if (threadIdx.x == 0)
            s_odd[1] = again ? 1.f : 0.f;
    }
    __syncthreads();
    if (s_odd[1] != 0.f) {  // the same in every block of the cluster
        const float w = s_weight[my_head * kMaxRanges + rank];
        const float inv = __fdiv_rn(1.f, s_total[my_head]);
        for (int i = threadIdx.x; i < n * HR; i += kAttnThreads)
            s_sc[i] = __fmul_rn(__fmul_rn(s_sc[i], w), inv);
        __syncthreads();  // scores final, weights read
        weigh_again(s_out);
        for (int i = threadIdx.x; i < HR * kMaxRanges; i += kAttnThreads)
            s_weight[i] = 1.f;
        if (threadIdx.x < HR)
            s_total[threadIdx.x] = 1.f;
        cluster.sync();
    }
    constexpr int kShare = HR * DIM / CTAS;  // outputs per block
    for (int u = threadIdx.x; u < kShare; u += kAttnThreads) {
        const int i = rank * kShare + u, h = i / DIM;
        float o[CTAS];
#pragma unroll
        for (int c = 0; c < CTAS; ++c)
            o[c] = cluster.map_shared_rank(s_out, c)[i];
        float a = 0.f;
#pragma unroll
        for (int c = 0; c < CTAS; ++c) {
            const float w = s_weight[h * kMaxRanges + c];
            if (w != 0.f)
                a = __fmaf_rn(w, o[c], a);
        }
        float l = s_total[h];  // NaN if any score was
        if (!(fabsf(a) <= FLT_MAX)) {  // finite sums that overflow together
            a = 0.f;
#pragma unroll 1
            for (int c = 0; c < CTAS; ++c) {
                const float w = __fdiv_rn(s_weight[h * kMaxRanges + c], l);
                if (w != 0.f)
                    a = __fmaf_rn(w, cluster.map_shared_rank(s_out, c)[i], a);
            }
            l = 1.f;
        }
        if (h < nh)
            out[row0 + i] = __fdiv_rn(a, l);
    }
    cluster.sync();  // nobody leaves while its sums may still be read
}

// A block per tile (attention_tile.cuh).
template <int DIM, int ROWS, bool ALIGNED>
__global__ void __launch_bounds__(kAttnThreads, DIM > 128 ? 1 : 2)
attention_tile_kernel(const float* __restrict__ q, const float* __restrict__ k_cache,
                      const float* __restrict__ v_cache, float* __restrict__ out, int tokens,
                      int heads, int kv_heads, int past0, const int* __restrict__ past_dev,
                      int capacity, float scale, int tq) {
    b2w4_pdl_chain_entry();
    const int past = past_dev ? min(*past_dev, capacity - tokens) : past0;
    extern __shared__ __align__(16) float s_dyn[];
    // the last tiles see the most keys: they go first, of all kv heads
    attention_tile<DIM, ROWS, ALIGNED, BlockSync>(
        q, k_cache, v_cache, out, tokens, heads, kv_heads, past, capacity, scale, tq, blockIdx.x,
        (int)(gridDim.y - 1 - blockIdx.y) * tq, s_dyn);
}

// A position counter on the device: *counter += by (after a decode step of a replayed graph),
// and the step's token appended to a history so that the host may read all of them at the end.
__global__ void advance_kernel(int* counter, int by, const int32_t* token, int32_t* history,
                               int history_len) {
    b2w4_pdl_chain_entry();
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const int at = *counter;
        if (history && token && at >= 0 && at < history_len)
            history[at] = *token;
        *counter = at + by;
    }
}

// OpType::CONTIGUOUS for a block of rows (kernels/layout.cpp materialises a strided view the
// same way): dst[r][c] = src[r][c], each side with its own row stride.
__global__ void copy_rows_kernel(const float* __restrict__ src, int ld_src,
                                 float* __restrict__ dst, int ld_dst, int rows, int cols) {
    b2w4_pdl_chain_entry();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols)
        return;
    const int r = (int)(i / cols), c = (int)(i - (size_t)r * cols);
    dst[(size_t)r * ld_dst + c] = src[(size_t)r * ld_src + c];
}

// Embedding lookup: rows of an fp16 table widened to fp32 (the reference's EMBEDDING input
// path widens fp16 rows the same way, engine/engine.cpp:637-672 uploads "hidden").
// One block per 1024 features of a row, four per thread (8-byte loads, 16-byte stores where the
// rows allow it); a thread per feature with 64-bit divisions took 18.5 us for 1500 rows of 2560.
constexpr int kEmbedThreads = 256;
__global__ void __launch_bounds__(kEmbedThreads)
embed_rows_kernel(const __half* __restrict__ table, const int32_t* __restrict__ ids, int dim,
                  float* __restrict__ out, int ldo, bool aligned) {
    b2w4_pdl_chain_entry();
    const int d = (blockIdx.y * kEmbedThreads + threadIdx.x) * 4;
    const __half* src = table + (size_t)ids[blockIdx.x] * dim + d;
    float* dst = out + (size_t)blockIdx.x * ldo + d;
    if (aligned && d < dim) {
        const uint2 raw = *reinterpret_cast<const uint2*>(src);
        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
        const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
        *reinterpret_cast<float4*>(dst) = make_float4(lo.x, lo.y, hi.x, hi.y);
    } else {
        for (int i = 0; i < 4 && d + i < dim; ++i)
            dst[i] = __half2float(src[i]);
    }
}

// ---- which kernel a call takes, and its launch ----
enum AttnForm { ATTN_ROW, ATTN_PLAIN, ATTN_SPLIT, ATTN_TILE };
struct AttnPlan {
    int form;
    int rows;       // ATTN_TILE: rows per tile
    int ctas;       // ATTN_SPLIT: blocks per cluster
    int one_range;  // ATTN_SPLIT: visible keys up to which one block takes them all
    bool alone;     // ATTN_TILE: one block per multiprocessor
};
struct AttnArgs {
    const float *q, *k_cache, *v_cache;
    float* out;
    int tokens, heads, kv_heads, past;
    const int* past_dev;
    int capacity;
    float scale;
    const PrepArgs* prep;  // the split kernel with one token: rows from the qkv matmul
};

// query heads of a kv head that a block of the split kernel serves
int split_heads(int dim, int rep) { return dim == 256 ? min(rep, 2) : rep >= 3 ? 4 : rep; }

// Time of the tile kernel with one block per multiprocessor, in the time of the largest tile
// (its last token sees past + tokens keys, the first tile's about past): one wave is as long as
// its largest tile; in a second one the largest tiles that are left go where the smallest of
// the first wave were, and all such pairs are equally long; beyond that the load counts.
double tile_blocks(int tokens, int rep, int rows, int kv_heads) {
    return rep > rows ? 1e9 : (double)((tokens + rows / rep - 1) / (rows / rep)) * kv_heads;
}
double tile_load(int tokens, int rep, int rows, int kv_heads, int past, int sms) {
    return tile_blocks(tokens, rep, rows, kv_heads) / sms * (past + 0.5 * tokens) / (past + tokens);
}
double tile_time(int tokens, int rep, int rows, int kv_heads, int past, int sms) {
    const double n = tile_blocks(tokens, rep, rows, kv_heads);
    if (n <= sms)
        return 1.0;
    if (n <= 2.0 * sms)
        return max(1.0, 2.0 * (1.0 - (double)tokens / (past + tokens) * sms / n));
    return tile_load(tokens, rep, rows, kv_heads, past, sms) + 0.3;
}

// A call's form depends on its sizes and the cache's capacity, not on the position, so that a
// position given by the host and one read on the device leave the same bits (the tile kernel's
// variants do, too, so those are chosen by `past`).  The lines, times on a B200:
//   few rows   `groups` blocks with all keys (one_range), or clusters that split them.  A
//              cluster costs 2 to 3 us, more where there are many; 32 / 8 heads of 128, one
//              block against clusters: one token, 64 keys 5.1 / 5.6 us, 160 keys 7.1 / 5.8; 16
//              tokens, 300 keys 12.6 / 15.7, 1000 keys 36 / 26.  The cluster sizes keep all of
//              them resident at once (`places`, short of the last): sixteen against eight, one
//              token, 6000 keys 21.4 / 32.2, seven tokens 71 / 60, with four 59; and behind 300
//              keys eight are enough, one token 6.9 / 5.9.
//   up to      10 groups per multiprocessor; against the tile kernel: 32 / 8 heads of 128, 100
//              tokens behind 300 keys 41 / 57 us, 256 tokens 108 / 108; 16 / 8 heads of 64, 160
//              tokens 36 / 42, 256 tokens 56 / 49.
//   from       a capacity of 384 for runs of eight or more: below that the tile kernel is at
//              most some tens of us long, and keeps the bits of the one-row arithmetic.
//   unaligned  one block per (token, head) up to five per multiprocessor, then tiles: 32 / 8
//              heads of 128, 8 tokens behind 6000 keys 430 / 830 us, 32 tokens 910 / 840.
//   tiles      of 32 rows alone on a multiprocessor, of 64 alone (1.41 times as long), or two of
//              64 (1.6 times that, 0.82 of it per tile), by tile_time: 600 tokens of 32 / 8
//              heads 178 / 134 / 174 us, 1200 tokens 661 / 473 / 387, 256 tokens 39 / 52 / 62.
AttnPlan attn_plan(int tokens, int heads, int kv_heads, int dim, int past, int capacity,
                   bool aligned, bool row_only, int max_cluster, int sm_count) {
    const int rep = heads / kv_heads;
    AttnPlan p = {ATTN_ROW, 0, 0, 0, false};
    if (dim != 64 && dim != 128 && dim != 256)
        return p;
    if (row_only) {
        p.form = ATTN_PLAIN;
        return p;
    }
    const int hr = split_heads(dim, rep);
    const long groups = (long)tokens * kv_heads * ((rep + hr - 1) / hr);
    if (aligned && groups / tokens <= 65535 &&
        (tokens < 8 || (capacity >= 384 && groups <= 10l * sm_count))) {
        p.form = ATTN_SPLIT;
        const long places = (long)split_blocks(dim, hr) * sm_count;
        p.ctas = capacity >= 768 && groups * 16 * 5 <= places * 4 ? 16
                 : groups * 8 * 10 <= places * 9                  ? 8
                                                                  : 4;
        p.one_range = (int)min(4096l, max(p.ctas == 16 ? 96l : 128l, groups * groups / 32));
        while (p.ctas > max_cluster)
            p.ctas /= 2;
        return p;
    }
    if (rep > 64 || tokens < 8 || (!aligned && (long)tokens * heads <= 5l * sm_count))
        return p;
    p.form = ATTN_TILE;
    const double whole32 = tile_time(tokens, rep, 32, kv_heads, past, sm_count);
    const double whole64 = 1.41 * tile_time(tokens, rep, 64, kv_heads, past, sm_count);
    const double shared64 =
        1.41 * max(1.6, 0.82 * tile_load(tokens, rep, 64, kv_heads, past, sm_count));
    p.rows = whole32 <= min(whole64, shared64) ? 32 : 64;
    p.alone = p.rows == 32 || whole64 <= shared64;
    return p;
}

// Runs of tiles that take the tensor-core kernel (aligned rows), by what does not depend on the
// position: a cache of 384 rows (below that the one-row arithmetic's bits are kept, see above) and
// enough (token, head) rows for its blocks of 128 to fill a part of the chip.  Where it is taken it
// is closer to 64 bits than the tile kernel, and faster but for the shortest runs at the head of a
// cache; us, and error in 2-norm on normal inputs:
//   32 / 8 heads of 128   200 tokens 33.2 -> 35.3 (1.6e-7 -> 1.5e-7), 256 39.7 -> 34.7, behind 300
//                         keys 111 -> 59 (4.0e-7 -> 2.2e-7), 1500 589 -> 214 (3.1e-7 -> 1.8e-7),
//                         2000 behind 6000 keys 7074 -> 2172 (1.5e-6 -> 3.1e-7)
//   28 / 4 heads of 128   333 tokens behind 50 keys 77 -> 52; 64 / 1 heads, 129 behind 300 87 -> 51
//   64 / 8 heads of 64    380 tokens 76 -> 34, 1500 676 -> 277
// Error on other inputs, 32 / 8 heads, 256 tokens and 1500: values of one sign 1.8e-7 -> 0.8e-7 and
// 4.1e-7 -> 1.0e-7; scores thirty times as large 6.9e-7 -> 5.3e-7 and 9.3e-7 -> 7.7e-7; queries and
// values with the tails of exp(normal) 2.3e-7 -> 3.0e-7 and 5.8e-7 -> 3.4e-7 (the one kind of input
// on which short runs lose: sums in tensor memory truncate).
// The lines of rows per multiprocessor are not those of speed (8 / 8 heads of 128, 600 tokens behind
// 100 keys take 95 in tiles; 32 / 8 heads of 64, 640 tokens 97): shorter runs keep their bits.
bool attn_tensor(int tokens, int heads, int dim, int capacity, int sm_count) {
    return capacity >= 384 && (dim == 128 || dim == 64) &&
           (long)tokens * heads >= (dim == 128 ? 40l : 160l) * sm_count;
}

// Clusters of the kernel that the device holds at once (a slice of it may not have sixteen, or
// eight, multiprocessors side by side).
constexpr size_t kMaxBlockSmem = 220 * 1024;
// more dynamic shared memory than this, and a multiprocessor holds one block
constexpr size_t kHalfSmem = 114 * 1024;
template <typename Kernel>
int clusters_held(Kernel kern, int ctas, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kAttnThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = ctas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0)
        return n;
    (void)cudaGetLastError();
    return 0;
}

template <int DIM, int HR, int CTAS, bool PREP, bool RING>
int launch_split_as(b2w4_ctx* ctx, const AttnArgs& a, int keys, const AttnPlan& plan,
                    bool* placed) {
    static b2w4_smem_optin cfg, wide;
    static b2w4_smem_optin held;  // clusters_held + 1, per device
    auto kern = attention_split_kernel<DIM, HR, CTAS, PREP, RING>;
    const PrepArgs prep = PREP ? *a.prep : PrepArgs();
    const int range = max((keys + CTAS - 1) / CTAS, min(keys, plan.one_range));
    size_t smem = sizeof(float) * (SplitSmem<DIM, HR>::kScores + (size_t)range * HR);
    if (RING)
        smem += 128 + kAttnWarps * kRingSlots * kSlotBytes;
    const dim3 grid(CTAS, a.kv_heads * ((a.heads / a.kv_heads + HR - 1) / HR), a.tokens);
    if (smem > (RING ? kHalfSmem : kMaxBlockSmem))
        return B2W4_OK;  // not placed
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, RING ? kHalfSmem + 1 : smem, cfg));
    if constexpr (CTAS > 1)
        B2W4_CUDA(ctx, b2w4_opt_in_cluster(ctx, kern, wide));
    // a ring: asked with the most that its launch may take
    long clusters = 0;
    if (CTAS > 1) {
        size_t& n = held.bytes[ctx->device];
        if (!n)
            n = 1 + clusters_held(kern, CTAS, RING ? kHalfSmem + 1 : 32 * 1024);
        clusters = (long)n - 1;
        if (!clusters)
            return B2W4_OK;  // without a ring, or a smaller cluster
    }
    // A ring's blocks go to a multiprocessor each where all their clusters fit that way (sixteen
    // blocks of eight clusters do not: two waves, 33 us instead of 22).  A step of eight layers
    // behind 300 keys 317 -> 310 us.
    if (RING && (CTAS == 1 || clusters >= (long)grid.y * grid.z))
        smem = kHalfSmem + 1;
    if constexpr (CTAS == 1) {
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, grid, dim3(kAttnThreads), smem,
                                           ctx->stream, a.q, a.k_cache, a.v_cache, a.out,
                                           a.tokens, a.heads, a.kv_heads, a.past, a.past_dev,
                                           a.capacity, a.scale, plan.one_range, prep));
    } else {
        B2W4_CUDA(ctx, b2w4_launch_chained_cluster(
                           ctx->pdl, kern, grid, dim3(kAttnThreads), CTAS, smem, ctx->stream,
                           a.q, a.k_cache, a.v_cache, a.out, a.tokens, a.heads, a.kv_heads,
                           a.past, a.past_dev, a.capacity, a.scale, plan.one_range, prep));
    }
    ctx->launches++;
    *placed = true;
    return B2W4_OK;
}
template <int DIM, int HR, int CTAS>
int launch_split_ctas(b2w4_ctx* ctx, const AttnArgs& a, int keys, const AttnPlan& plan,
                      bool* placed) {
    if (!a.prep)
        return launch_split_as<DIM, HR, CTAS, false, false>(ctx, a, keys, plan, placed);
    // a decode step's blocks that have a multiprocessor each; scores that leave no room for the
    // ring take the launch without it
    if constexpr (DIM <= 128) {
        const int sets = (a.heads / a.kv_heads + HR - 1) / HR;
        if ((long)CTAS * a.kv_heads * sets <= ctx->sm_count) {
            const int rc = launch_split_as<DIM, HR, CTAS, true, true>(ctx, a, keys, plan, placed);
            if (rc != B2W4_OK || *placed)
                return rc;
        }
    }
    return launch_split_as<DIM, HR, CTAS, true, false>(ctx, a, keys, plan, placed);
}
// The planned cluster, or the next smaller one that the device can place.
template <int DIM, int HR>
int launch_split_hr(b2w4_ctx* ctx, const AttnArgs& a, int keys, const AttnPlan& plan,
                    bool* placed) {
    if (keys <= plan.one_range)
        return launch_split_ctas<DIM, HR, 1>(ctx, a, keys, plan, placed);
    int rc = B2W4_OK;
    if (plan.ctas >= 16)
        rc = launch_split_ctas<DIM, HR, 16>(ctx, a, keys, plan, placed);
    if (rc == B2W4_OK && !*placed && plan.ctas >= 8)
        rc = launch_split_ctas<DIM, HR, 8>(ctx, a, keys, plan, placed);
    if (rc == B2W4_OK && !*placed && plan.ctas >= 4)
        rc = launch_split_ctas<DIM, HR, 4>(ctx, a, keys, plan, placed);
    return rc;
}

int launch_split(b2w4_ctx* ctx, const AttnArgs& a, int dim, int keys, const AttnPlan& plan,
                 bool* placed) {
    const int hr = split_heads(dim, a.heads / a.kv_heads);
    switch (dim * 8 + hr) {
    case 64 * 8 + 1: return launch_split_hr<64, 1>(ctx, a, keys, plan, placed);
    case 64 * 8 + 2: return launch_split_hr<64, 2>(ctx, a, keys, plan, placed);
    case 64 * 8 + 4: return launch_split_hr<64, 4>(ctx, a, keys, plan, placed);
    case 128 * 8 + 1: return launch_split_hr<128, 1>(ctx, a, keys, plan, placed);
    case 128 * 8 + 2: return launch_split_hr<128, 2>(ctx, a, keys, plan, placed);
    case 128 * 8 + 4: return launch_split_hr<128, 4>(ctx, a, keys, plan, placed);
    case 256 * 8 + 1: return launch_split_hr<256, 1>(ctx, a, keys, plan, placed);
    default: return launch_split_hr<256, 2>(ctx, a, keys, plan, placed);
    }
}

template <int DIM, int ROWS, bool ALIGNED>
int launch_tile_as(b2w4_ctx* ctx, const AttnArgs& a, bool alone) {
    static b2w4_smem_optin cfg;
    auto kern = attention_tile_kernel<DIM, ROWS, ALIGNED>;
    const int tq = ROWS / (a.heads / a.kv_heads);
    const dim3 grid(a.kv_heads, (a.tokens + tq - 1) / tq);
    const size_t smem = max((size_t)TileSmem<DIM, ROWS>::kBytes, alone ? kHalfSmem + 1 : 0);
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, cfg));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, grid, dim3(kAttnThreads), smem,
                                       ctx->stream, a.q, a.k_cache, a.v_cache, a.out, a.tokens,
                                       a.heads, a.kv_heads, a.past, a.past_dev, a.capacity,
                                       a.scale, tq));
    ctx->launches++;
    return B2W4_OK;
}
template <int DIM>
int launch_tile_dim(b2w4_ctx* ctx, const AttnArgs& a, const AttnPlan& plan, bool aligned) {
    if (plan.rows == 32)
        return aligned ? launch_tile_as<DIM, 32, true>(ctx, a, plan.alone)
                       : launch_tile_as<DIM, 32, false>(ctx, a, plan.alone);
    return aligned ? launch_tile_as<DIM, 64, true>(ctx, a, plan.alone)
                   : launch_tile_as<DIM, 64, false>(ctx, a, plan.alone);
}
int launch_tile(b2w4_ctx* ctx, const AttnArgs& a, int dim, const AttnPlan& plan, bool aligned) {
    return dim == 64    ? launch_tile_dim<64>(ctx, a, plan, aligned)
           : dim == 128 ? launch_tile_dim<128>(ctx, a, plan, aligned)
                        : launch_tile_dim<256>(ctx, a, plan, aligned);
}

}  // namespace

int b2w4_launch_step_norm(b2w4_ctx* ctx, const b2w4_norm_args& n, int k, float* hidden) {
    if (!n.update && n.residual_out)  // first: hidden may be the residual itself
        B2W4_CUDA(ctx, cudaMemcpyAsync(n.residual_out, n.residual, sizeof(float) * k,
                                       cudaMemcpyDeviceToDevice, ctx->stream));
    if (!n.update)
        return b2w4_rms_norm(ctx, n.residual, k, 1, k, n.weight, n.eps, hidden, k);
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, rms_norm_kernel, dim3(1), dim3(kNormThreads), 0,
                                       ctx->stream, n.residual, k, n.update, k, n.residual_out, k,
                                       n.weight, n.eps, hidden, k));
    ctx->launches++;
    return B2W4_OK;
}

extern "C" {

int b2w4_rms_norm(b2w4_ctx* ctx, const float* x_dev, int ldx, int rows, int dim,
                  const float* weight_dev, float eps, float* out_dev, int ldo) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!x_dev || !weight_dev || !out_dev || rows <= 0 || dim <= 0 || ldx < dim || ldo < dim)
        return b2w4_fail(ctx, B2W4_E_INVALID, "rms_norm: bad argument");
    if (dim <= kNormWarpMaxK) {
        const size_t threads = (size_t)rows * 32;
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, rms_norm_warp_kernel,
                                           dim3((unsigned)((threads + 255) / 256)), dim3(256), 0,
                                           ctx->stream, x_dev, ldx, rows, dim, weight_dev, eps,
                                           out_dev, ldo));
    } else {
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, rms_norm_kernel, dim3(rows),
                                           dim3(kNormThreads), 0, ctx->stream,
                                           x_dev, ldx, static_cast<const float*>(nullptr), 0,
                                           static_cast<float*>(nullptr), dim, weight_dev, eps,
                                           out_dev, ldo));
    }
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_add_rms_norm(b2w4_ctx* ctx, float* residual_dev, int ldr, const float* update_dev,
                      int ldu, int rows, int dim, const float* weight_dev, float eps,
                      float* out_dev, int ldo) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!residual_dev || !update_dev || !weight_dev || !out_dev || rows <= 0 || dim <= 0 ||
        ldr < dim || ldu < dim || ldo < dim)
        return b2w4_fail(ctx, B2W4_E_INVALID, "add_rms_norm: bad argument");
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, rms_norm_kernel, dim3(rows), dim3(kNormThreads), 0,
                                       ctx->stream, residual_dev, ldr, update_dev, ldu,
                                       residual_dev, dim, weight_dev, eps, out_dev, ldo));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_swiglu(b2w4_ctx* ctx, const float* merged_dev, int ldm, int rows, int intermediate,
                float* out_dev, int ldo) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!merged_dev || !out_dev || rows <= 0 || intermediate <= 0 || ldm < 2 * intermediate ||
        ldo < intermediate)
        return b2w4_fail(ctx, B2W4_E_INVALID, "swiglu: bad argument");
    const size_t n = (size_t)rows * intermediate;
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, swiglu_kernel, dim3((unsigned)((n + 255) / 256)),
                                       dim3(256), 0, ctx->stream, merged_dev, ldm, rows,
                                       intermediate, out_dev, ldo));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_elementwise(b2w4_ctx* ctx, const float* a_dev, const float* b_dev, float* out_dev,
                     size_t count, int multiply) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!a_dev || !b_dev || !out_dev || count == 0)
        return b2w4_fail(ctx, B2W4_E_INVALID, "elementwise: bad argument");
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, binary_kernel,
                                       dim3((unsigned)((count + 255) / 256)), dim3(256), 0,
                                       ctx->stream, a_dev, b_dev, out_dev, count, multiply));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_rope(b2w4_ctx* ctx, const float* x_dev, float* out_dev, int tokens, int heads, int dim,
              const float* cos_dev, const float* sin_dev, int rope_dim, int first_position,
              const int* position_dev) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!x_dev || !out_dev || !cos_dev || !sin_dev || tokens <= 0 || heads <= 0 || dim <= 0 ||
        rope_dim <= 0 || rope_dim > dim || (rope_dim & 1) || first_position < 0)
        return b2w4_fail(ctx, B2W4_E_INVALID, "rope: bad argument");
    const size_t n = (size_t)tokens * heads * ((size_t)rope_dim / 2 + (dim - rope_dim));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, rope_kernel, dim3((unsigned)((n + 255) / 256)),
                                       dim3(256), 0, ctx->stream, x_dev, out_dev, tokens, heads,
                                       dim, cos_dev, sin_dev, rope_dim, first_position,
                                       position_dev));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_attention(b2w4_ctx* ctx, const float* q_dev, const float* k_dev, const float* v_dev,
                   float* k_cache_dev, float* v_cache_dev, float* out_dev, int tokens, int heads,
                   int kv_heads, int dim, int past, const int* past_dev, int capacity,
                   float scale) {
    if (!ctx)
        return B2W4_E_INVALID;
    const bool append = k_dev || v_dev;  // neither: the cache rows are in place already
    if (!q_dev || (append && (!k_dev || !v_dev)) || !k_cache_dev || !v_cache_dev || !out_dev ||
        tokens <= 0 || heads <= 0 || kv_heads <= 0 || heads % kv_heads || dim <= 0 ||
        dim > kAttnMaxDim || past < 0 || past + tokens > capacity)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "attention: bad argument (tokens=%d past=%d capacity=%d heads=%d/%d)",
                         tokens, past, capacity, heads, kv_heads);
    const int keys = past_dev ? capacity : past + tokens;  // position on the device: sized
                                                           // for a full cache
    const bool aligned = !(((uintptr_t)q_dev | (uintptr_t)k_cache_dev | (uintptr_t)v_cache_dev |
                            (uintptr_t)out_dev) & 15);
    auto plan_for = [&](int cap) {
        return attn_plan(tokens, heads, kv_heads, dim, past_dev ? capacity - tokens : past, cap,
                         aligned, !ctx->attn_tiles, ctx->attn_cluster, ctx->sm_count);
    };
    AttnPlan plan = plan_for(capacity);
    const int score_slots = (keys + 3) & ~3;
    if (sizeof(float) * ((size_t)score_slots + kAttnStage) > 200 * 1024)
        return b2w4_fail(ctx, B2W4_E_INVALID, "attention: %d keys exceed the score buffer", keys);
    if (append) {
        const size_t n = (size_t)tokens * kv_heads * dim;
        B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kv_append_kernel,
                                           dim3((unsigned)((n + 255) / 256)), dim3(256), 0,
                                           ctx->stream, k_dev, v_dev, k_cache_dev, v_cache_dev,
                                           tokens, kv_heads, dim, past, past_dev, capacity));
        ctx->launches++;
    }
    const AttnArgs a = {q_dev, k_cache_dev, v_cache_dev, out_dev, tokens, heads, kv_heads, past,
                        past_dev, capacity, scale, nullptr};
    if (plan.form == ATTN_SPLIT) {
        bool placed = false;
        const int rc = launch_split(ctx, a, dim, keys, plan, &placed);
        if (rc != B2W4_OK || placed)
            return rc;
        plan = plan_for(0);  // no cluster fits: runs as on a small cache, few tokens by row
    }
    if (plan.form == ATTN_TILE) {
        if (aligned && attn_tensor(tokens, heads, dim, capacity, ctx->sm_count))
            return b2w4_launch_attention_tc(ctx, q_dev, k_cache_dev, v_cache_dev, out_dev, tokens,
                                            heads, kv_heads, dim, past, past_dev, capacity, scale);
        return launch_tile(ctx, a, dim, plan, aligned);
    }
    static b2w4_smem_optin configured[2];
    const bool plain = plan.form == ATTN_PLAIN;
    auto kern = plain ? attention_plain_kernel : attention_kernel;
    const size_t row_smem =
        sizeof(float) *
        ((size_t)score_slots + (plain ? (keys + kTileKeys - 1) / kTileKeys : kAttnStage));
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, row_smem, configured[plain]));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, dim3(tokens * heads), dim3(kAttnThreads),
                                       row_smem, ctx->stream, q_dev, k_cache_dev, v_cache_dev,
                                       out_dev, tokens, heads, kv_heads, dim, past, past_dev,
                                       capacity, scale, score_slots));
    ctx->launches++;
    return B2W4_OK;
}

// What attn_plan says, for checks without a device: the form; out: rows, ctas, one_range, alone.
int b2w4_attention_plan(int tokens, int heads, int kv_heads, int dim, int past, int capacity,
                        int aligned, int row_only, int max_cluster, int sm_count, int* out) {
    const AttnPlan p = attn_plan(tokens, heads, kv_heads, dim, past, capacity, aligned, row_only,
                                 max_cluster, sm_count);
    out[0] = p.rows;
    out[1] = p.ctas;
    out[2] = p.one_range;
    out[3] = p.alone;
    return p.form;
}

int b2w4_qkv_prepare(b2w4_ctx* ctx, const float* qkv_dev, int ld, int tokens, int heads,
                     int kv_heads, int dim, const float* q_weight_dev, const float* k_weight_dev,
                     float eps, const float* cos_dev, const float* sin_dev, int past,
                     const int* past_dev, float* q_out_dev, float* k_cache_dev, float* v_cache_dev,
                     int capacity) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!qkv_dev || !cos_dev || !sin_dev || !q_out_dev || !k_cache_dev || !v_cache_dev ||
        tokens <= 0 || heads <= 0 || kv_heads <= 0 || dim <= 0 || dim > kAttnMaxDim || dim % 64 ||
        ld < (heads + 2 * kv_heads) * dim || past < 0 || past + tokens > capacity)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "qkv_prepare: bad argument (tokens=%d past=%d capacity=%d dim=%d)", tokens,
                         past, capacity, dim);
    auto kern = dim == 64    ? qkv_prepare_kernel<64>
                : dim == 128 ? qkv_prepare_kernel<128>
                : dim == 192 ? qkv_prepare_kernel<192>
                             : qkv_prepare_kernel<256>;
    const size_t warps = (size_t)tokens * (heads + 2 * kv_heads);
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern, dim3((unsigned)((warps + 7) / 8)),
                                       dim3(256), 0, ctx->stream, qkv_dev, ld, (unsigned)tokens,
                                       heads, kv_heads, q_weight_dev, k_weight_dev, eps, cos_dev,
                                       sin_dev, past, past_dev, q_out_dev, k_cache_dev,
                                       v_cache_dev, capacity));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_attention_step(b2w4_ctx* ctx, const float* qkv_dev, int heads, int kv_heads, int dim,
                        const float* q_weight_dev, const float* k_weight_dev, float eps,
                        const float* cos_dev, const float* sin_dev, int past, const int* past_dev,
                        float* q_work_dev, float* k_cache_dev, float* v_cache_dev, float* out_dev,
                        int capacity, float scale) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!qkv_dev || !cos_dev || !sin_dev || !q_work_dev || !k_cache_dev || !v_cache_dev ||
        !out_dev || heads <= 0 || kv_heads <= 0 || heads % kv_heads || dim <= 0 ||
        dim > kAttnMaxDim || dim % 64 || past < 0 || past + 1 > capacity)
        return b2w4_fail(ctx, B2W4_E_INVALID,
                         "attention_step: bad argument (past=%d capacity=%d heads=%d/%d dim=%d)",
                         past, capacity, heads, kv_heads, dim);
    const int keys = past_dev ? capacity : past + 1;
    const bool aligned = !(((uintptr_t)k_cache_dev | (uintptr_t)v_cache_dev |
                            (uintptr_t)out_dev) & 15);
    const AttnPlan plan = attn_plan(1, heads, kv_heads, dim, past_dev ? capacity - 1 : past,
                                    capacity, aligned, !ctx->attn_tiles, ctx->attn_cluster,
                                    ctx->sm_count);
    // out over the rows: blocks would store it while others still read theirs
    const bool apart = !b2w4_overlap(out_dev, sizeof(float) * heads * dim, qkv_dev,
                                     sizeof(float) * (heads + 2 * kv_heads) * dim);
    // the refusal of long caches is b2w4_attention's, in every form
    if (apart && plan.form == ATTN_SPLIT &&
        sizeof(float) * (((keys + 3) & ~3) + kAttnStage) <= 200 * 1024) {
        const PrepArgs prep = {qkv_dev, q_weight_dev, k_weight_dev, cos_dev, sin_dev,
                               eps,     k_cache_dev,  v_cache_dev};
        const AttnArgs a = {nullptr, k_cache_dev, v_cache_dev, out_dev,  1,     heads,
                            kv_heads, past,       past_dev,    capacity, scale, &prep};
        bool placed = false;
        const int rc = launch_split(ctx, a, dim, keys, plan, &placed);
        if (rc != B2W4_OK || placed)
            return rc;
    }
    const int rc = b2w4_qkv_prepare(ctx, qkv_dev, (heads + 2 * kv_heads) * dim, 1, heads,
                                    kv_heads, dim, q_weight_dev, k_weight_dev, eps, cos_dev,
                                    sin_dev, past, past_dev, q_work_dev, k_cache_dev, v_cache_dev,
                                    capacity);
    if (rc != B2W4_OK)
        return rc;
    return b2w4_attention(ctx, q_work_dev, nullptr, nullptr, k_cache_dev, v_cache_dev, out_dev, 1,
                          heads, kv_heads, dim, past, past_dev, capacity, scale);
}

int b2w4_advance(b2w4_ctx* ctx, int* counter_dev, int by, const int32_t* token_dev,
                 int32_t* history_dev, int history_len) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!counter_dev)
        return b2w4_fail(ctx, B2W4_E_INVALID, "advance: no counter");
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, advance_kernel, dim3(1), dim3(32), 0, ctx->stream,
                                       counter_dev, by, token_dev, history_dev, history_len));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_copy_rows(b2w4_ctx* ctx, const float* src_dev, int ld_src, float* dst_dev, int ld_dst,
                   int rows, int cols) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!src_dev || !dst_dev || rows <= 0 || cols <= 0 || ld_src < cols || ld_dst < cols)
        return b2w4_fail(ctx, B2W4_E_INVALID, "copy_rows: bad argument");
    const size_t n = (size_t)rows * cols;
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, copy_rows_kernel,
                                       dim3((unsigned)((n + 255) / 256)), dim3(256), 0,
                                       ctx->stream, src_dev, ld_src, dst_dev, ld_dst, rows, cols));
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_embed_rows(b2w4_ctx* ctx, const void* table_fp16_dev, const int32_t* ids_dev, int rows,
                    int dim, float* out_dev, int ldo) {
    if (!ctx)
        return B2W4_E_INVALID;
    if (!table_fp16_dev || !ids_dev || !out_dev || rows <= 0 || dim <= 0 || ldo < dim)
        return b2w4_fail(ctx, B2W4_E_INVALID, "embed_rows: bad argument");
    const bool aligned = !(((uintptr_t)table_fp16_dev & 7) | ((uintptr_t)out_dev & 15) |
                           (dim & 3) | (ldo & 3));
    const int per_block = 4 * kEmbedThreads;
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, embed_rows_kernel,
                                       dim3(rows, (dim + per_block - 1) / per_block),
                                       dim3(kEmbedThreads), 0, ctx->stream,
                                       static_cast<const __half*>(table_fp16_dev), ids_dev, dim,
                                       out_dev, ldo, aligned));
    ctx->launches++;
    return B2W4_OK;
}

}  // extern "C"
