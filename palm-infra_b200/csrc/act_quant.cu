// Stand-alone activation quantiser: fp32 rows -> int8 codes + one fp32 scale per group.
// Follows the reference quantisers' rounding points exactly
// (kernels/matmul_quant.cpp:578-641 per 128 values, :280-329 per 32 values): amax over the
// group, scale = amax/127 (1 when amax == 0), codes = clamp(rint(x * (127/amax)), +-127).
#include "b200w4_internal.cuh"

namespace {

// one warp per (row, 128-group); lane holds k = 4*lane .. 4*lane+3 of the group
template <int RULE, int LAYOUT>
__global__ void quantize_rows_kernel(const float* __restrict__ x, int lda, int m, int k,
                                     int8_t* __restrict__ q, float* __restrict__ scales) {
    b2w4_pdl_chain_entry();
    const int groups = k >> 7;
    long long wid = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wid >= (long long)m * groups)
        return;
    const int row = (int)(wid / groups), g = (int)(wid % groups);
    const float* src = x + (size_t)row * lda + (size_t)g * 128 + lane * 4;
    float v0 = src[0], v1 = src[1], v2 = src[2], v3 = src[3];
    float amax = fmaxf(fmaxf(fabsf(v0), fabsf(v1)), fmaxf(fabsf(v2), fabsf(v3)));
    // max is exact and order-free, so a butterfly gives the sequential loop's value
    const int span = RULE == 128 ? 32 : 8;
#pragma unroll
    for (int off = span / 2; off > 0; off >>= 1)
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    float scale, inv;
    b2w4_quant_params(amax, scale, inv);
    const int c0 = b2w4_quant_code(v0, inv), c1 = b2w4_quant_code(v1, inv);
    const int c2 = b2w4_quant_code(v2, inv), c3 = b2w4_quant_code(v3, inv);
    if (RULE == 128) {
        if (lane == 0)
            scales[(size_t)row * groups + g] = scale;
    } else if ((lane & 7) == 0) {
        scales[(size_t)row * (groups * 4) + g * 4 + (lane >> 3)] = scale;
    }
    int8_t* dst = q + (size_t)row * k + (size_t)g * 128;
    if (LAYOUT == QLAYOUT_NATURAL) {
        char4 packed = make_char4((signed char)c0, (signed char)c1, (signed char)c2,
                                  (signed char)c3);
        *reinterpret_cast<char4*>(dst + lane * 4) = packed;
    } else {
        // 32-block `sub` = lane/8 stored as 16 even-k codes then 16 odd-k codes
        int8_t* blk = dst + (lane >> 3) * 32;
        const int j = (lane & 7) * 2;
        *reinterpret_cast<char2*>(blk + j) = make_char2((signed char)c0, (signed char)c2);
        *reinterpret_cast<char2*>(blk + 16 + j) =
            make_char2((signed char)c1, (signed char)c3);
    }
}

// ---- quantisers of the many-row matmuls -------------------------------------------------------
// What a quantised row is laid out for:
//   UMMA   the tensor-core kernels: per 128-k group a plane of [m_pad rows][128 bytes]; inside a
//          row's 128 bytes the 32-block `sub` is the 16-byte chunk pair (2*sub: even k, 2*sub+1:
//          odd k), and chunk c is stored at position c ^ (row % 8): the 128-byte swizzle the
//          MMA's shared-memory descriptor expects, so the plane can be bulk-copied into shared
//          memory as is.  Scales: fp32 [groups][m_pad]; with one scale per 32 values (A32)
//          [groups][m_pad][4], a row's four block scales side by side
//   MMA    the mma.sync GEMM: codes int8 [m][K] in tensor-operand order (inside a 128-group
//          [word position p 0..3][32 bytes]: the even-k codes 4p..4p+3 of the four 32-blocks, then
//          the odd ones, so that the B words of a lane of m16n8k32 are contiguous), scales and
//          the accumulator bias 0x4B400000 - 8 * (sum of the group's codes) transposed to
//          [groups][m_pad] (A32: [groups*4][m_pad], one entry per 32-block) so that one group of
//          all rows is contiguous.  (The kernel multiplies unsigned nibbles q+8; starting its
//          int32 accumulator at the bias makes it end as 0x4B400000 + D, the bit pattern of the
//          float 12582912 + D.)
//   ROWS   the kernel for a few rows: codes as MMA, scales [groups][m_pad] (A32: [groups]
//          [m_pad / 2][4][2], a row pair's block scales side by side), no biases
enum { OUT_UMMA, OUT_MMA, OUT_ROWS };
struct QuantOut {
    int8_t* q;
    float* scales;
    int32_t* es;  // MMA
    int k, m_pad;
};

// One warp: a group of a row, lane l holds its values 4*l..+3.
template <int OUT, bool A32>
__device__ __forceinline__ void quantize_group(const QuantOut& o, int row, int g, int lane,
                                               const float (&v)[4]) {
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
    // per 128 values: all 32 lanes; per 32 values: the 8 lanes of a 32-block
#pragma unroll
    for (int off = A32 ? 4 : 16; off > 0; off >>= 1)
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, off));
    float scale, inv;
    b2w4_quant_params(amax, scale, inv);
    const int c0 = b2w4_quant_code(v[0], inv), c1 = b2w4_quant_code(v[1], inv);
    const int c2 = b2w4_quant_code(v[2], inv), c3 = b2w4_quant_code(v[3], inv);
    const char2 even = make_char2((signed char)c0, (signed char)c2);
    const char2 odd = make_char2((signed char)c1, (signed char)c3);
    const int sub = lane >> 3;  // 32-block
    const bool first = A32 ? (lane & 7) == 0 : lane == 0;
    if (OUT == OUT_UMMA) {
        if (first)
            o.scales[A32 ? ((size_t)g * o.m_pad + row) * 4 + sub : (size_t)g * o.m_pad + row] =
                scale;
        int8_t* rowp = o.q + ((size_t)g * o.m_pad + row) * 128;
        const int j = (lane & 7) * 2, sw = row & 7;
        *reinterpret_cast<char2*>(rowp + (((2 * sub) ^ sw) << 4) + j) = even;
        *reinterpret_cast<char2*>(rowp + (((2 * sub + 1) ^ sw) << 4) + j) = odd;
        return;
    }
    if (OUT == OUT_MMA) {
        int esum = c0 + c1 + c2 + c3;  // integer: order-free
#pragma unroll
        for (int off = A32 ? 4 : 16; off > 0; off >>= 1)
            esum += __shfl_xor_sync(0xffffffffu, esum, off);
        if (first) {
            const size_t at = (size_t)(A32 ? g * 4 + sub : g) * o.m_pad + row;
            o.scales[at] = scale;
            o.es[at] = 0x4B400000 - 8 * esum;
        }
    } else if (first) {
        o.scales[A32 ? (size_t)g * 4 * o.m_pad + (row >> 1) * 8 + sub * 2 + (row & 1)
                     : (size_t)g * o.m_pad + row] = scale;
    }
    // the lane's codes: even-k indices 2*(lane%8) and +1 of its 32-block, and the odd ones
    int8_t* blk = o.q + (size_t)row * o.k + (size_t)g * 128 + ((lane & 7) >> 1) * 32 + sub * 4 +
                  (lane & 1) * 2;
    *reinterpret_cast<char2*>(blk) = even;
    *reinterpret_cast<char2*>(blk + 16) = odd;
}

__device__ __forceinline__ void load4(const float* p, bool aligned, float (&v)[4]) {
    if (aligned) {
        const float4 f = *reinterpret_cast<const float4*>(p);
        v[0] = f.x, v[1] = f.y, v[2] = f.z, v[3] = f.w;
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = p[i];
    }
}
__device__ __forceinline__ bool rows_aligned(const float* p, int ld) {
    return ((reinterpret_cast<uintptr_t>(p) & 15) | (ld & 3)) == 0;
}

// Rows as they are, or (SWIGLU) SwiGLU of merged rows [2K] = gate | up with the operations of
// b2w4_swiglu, so that its result is not written and read again.  One warp per (row, group);
// indices in 32 bits, a 64-bit division costs more than the rest.
template <int OUT, bool A32, bool SWIGLU>
__global__ void __launch_bounds__(256)
quantize_rows_many_kernel(const float* __restrict__ x, int lda, unsigned m, const QuantOut o) {
    b2w4_pdl_chain_entry();  // the GEMM behind may start fetching its weights
    const unsigned groups = (unsigned)o.k >> 7;
    const unsigned wid = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (wid >= m * groups)
        return;
    const unsigned row = wid / groups, g = wid - row * groups;
    const float* src = x + (size_t)row * lda + g * 128 + lane * 4;
    const bool aligned = rows_aligned(x, lda);
    float v[4];
    load4(src, aligned, v);
    if (SWIGLU) {
        float u[4];
        load4(src + o.k, aligned, u);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = b2w4_swiglu_value(v[i], u[i]);
    }
    quantize_group<OUT, A32>(o, (int)row, (int)g, lane, v);
}

// The residual add and RMSNorm in front of a matmul, quantised as they are made: one block per
// row, the normalised row is not written.  The bits of b2w4_add_rms_norm: a thread adds every
// 256th square; the row waits in shared memory to be taken up group by group.
constexpr int kNormThreads = 256;
template <int OUT, bool A32>
__global__ void __launch_bounds__(kNormThreads)
quantize_norm_kernel(float* __restrict__ residual, int ldr, const float* __restrict__ update,
                     int ldu, const float* __restrict__ weight, float eps, const QuantOut o) {
    b2w4_pdl_chain_entry();
    extern __shared__ __align__(16) float s_row[];
    __shared__ float s_part[kNormThreads / 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x;
    float* r = residual + (size_t)row * ldr;
    const float* u = update ? update + (size_t)row * ldu : nullptr;
    float ss = 0.f;
#pragma unroll 10
    for (int d = threadIdx.x; d < o.k; d += kNormThreads) {
        float v = r[d];
        if (u) {
            v = __fadd_rn(v, u[d]);
            r[d] = v;
        }
        s_row[d] = v;
        ss = __fadd_rn(ss, __fmul_rn(v, v));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        ss = __fadd_rn(ss, __shfl_xor_sync(0xffffffffu, ss, off));
    if (lane == 0)
        s_part[warp] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int w = 0; w < kNormThreads / 32; ++w)
        ss = __fadd_rn(ss, s_part[w]);
    const float rms = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(ss, (float)o.k), eps)));
    const bool wa = rows_aligned(weight, 0);
#pragma unroll 2
    for (int g = warp; g < o.k >> 7; g += kNormThreads / 32) {
        const int at = g * 128 + lane * 4;
        float v[4], w[4];
        load4(s_row + at, true, v);
        load4(weight + at, wa, w);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            v[i] = __fmul_rn(__fmul_rn(v[i], rms), w[i]);
        quantize_group<OUT, A32>(o, row, g, lane, v);
    }
}

template <int OUT, bool A32>
cudaError_t launch_quantize_many(b2w4_ctx* ctx, const float* x, int lda, int m, const QuantOut& o,
                                 const b2w4_rows* from) {
    if (from && from->kind == b2w4_rows::NORM)
        return b2w4_launch_chained(ctx->pdl, quantize_norm_kernel<OUT, A32>, dim3(m),
                                   dim3(kNormThreads), sizeof(float) * o.k, ctx->stream,
                                   from->residual,
                                   from->ld, from->update, from->ldu, from->weight, from->eps, o);
    const unsigned grid = (unsigned)(((long long)m * (o.k / 128) + 7) / 8);
    if (from)
        return b2w4_launch_chained(ctx->pdl, quantize_rows_many_kernel<OUT, A32, true>, dim3(grid),
                                   dim3(256), 0, ctx->stream, from->merged, from->ld, (unsigned)m,
                                   o);
    return b2w4_launch_chained(ctx->pdl, quantize_rows_many_kernel<OUT, A32, false>, dim3(grid),
                               dim3(256), 0, ctx->stream, x, lda, (unsigned)m, o);
}

}  // namespace

int b2w4_launch_quantize_mma(b2w4_ctx* ctx, const float* x, int lda, int m, int k, int m_pad,
                             int act_rule, int8_t* q, float* scales_t, int32_t* es_t) {
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (lda & 3))
        return b2w4_fail(ctx, B2W4_E_INVALID, "quantize: rows must be 16-byte aligned");
    const QuantOut o = {q, scales_t, es_t, k, m_pad};
    const cudaError_t e = act_rule == B2W4_ACT_G32
                              ? launch_quantize_many<OUT_MMA, true>(ctx, x, lda, m, o, nullptr)
                              : launch_quantize_many<OUT_MMA, false>(ctx, x, lda, m, o, nullptr);
    B2W4_CUDA(ctx, e);
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_launch_quantize_rows(b2w4_ctx* ctx, const float* x, int lda, int m, int k, int m_pad,
                              int act_rule, int8_t* q, float* scales, const b2w4_rows* from) {
    const QuantOut o = {q, scales, nullptr, k, m_pad};
    const cudaError_t e = act_rule == B2W4_ACT_G32
                              ? launch_quantize_many<OUT_ROWS, true>(ctx, x, lda, m, o, from)
                              : launch_quantize_many<OUT_ROWS, false>(ctx, x, lda, m, o, from);
    B2W4_CUDA(ctx, e);
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_launch_quantize_umma(b2w4_ctx* ctx, const float* x, int lda, int m, int k, int m_pad,
                              int act_rule, int8_t* q, float* scales, const b2w4_rows* from) {
    const QuantOut o = {q, scales, nullptr, k, m_pad};
    const cudaError_t e = act_rule == B2W4_ACT_G32
                              ? launch_quantize_many<OUT_UMMA, true>(ctx, x, lda, m, o, from)
                              : launch_quantize_many<OUT_UMMA, false>(ctx, x, lda, m, o, from);
    B2W4_CUDA(ctx, e);
    ctx->launches++;
    return B2W4_OK;
}

int b2w4_launch_quantize(b2w4_ctx* ctx, const float* x, int lda, int m, int k,
                         int act_rule, int8_t* q, float* scales, int layout) {
    if (k <= 0 || k % 128 != 0 || m <= 0 || lda < k)
        return b2w4_fail(ctx, B2W4_E_INVALID, "quantize: bad shape m=%d k=%d lda=%d", m,
                         k, lda);
    if (act_rule != B2W4_ACT_G128 && act_rule != B2W4_ACT_G32)
        return b2w4_fail(ctx, B2W4_E_INVALID, "quantize: act_rule must be 128 or 32");
    long long warps = (long long)m * (k / 128);
    int grid = (int)((warps * 32 + 255) / 256);
#define LAUNCH(R, L)                                                                         \
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, quantize_rows_kernel<R, L>, dim3(grid),        \
                                       dim3(256), 0, ctx->stream, x, lda, m, k, q, scales))
    if (act_rule == 128 && layout == QLAYOUT_NATURAL)
        LAUNCH(128, QLAYOUT_NATURAL);
    else if (act_rule == 128)
        LAUNCH(128, QLAYOUT_EVEN_ODD);
    else if (layout == QLAYOUT_NATURAL)
        LAUNCH(32, QLAYOUT_NATURAL);
    else
        LAUNCH(32, QLAYOUT_EVEN_ODD);
#undef LAUNCH
    ctx->launches++;
    B2W4_CUDA(ctx, cudaGetLastError());
    return B2W4_OK;
}
