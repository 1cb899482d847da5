// Attention of a tile of (token, head) rows on the fp32 pipe: shared by the kernel that takes
// tiles block by block (decoder_ops.cu) and by the tensor-core kernel for tiles whose sums come
// out not finite (attention_tc.cu).
#pragma once

#include "b200w4_internal.cuh"

namespace {

constexpr int kAttnThreads = 256;

// Softmax over blocks of kTileKeys keys in order: the running maximum m moves, and what is
// summed so far is scaled by exp(m_old - m_new).
constexpr int kTileKeys = 32;
__device__ __forceinline__ float attn_rescale(float m_old, float m_new) {
    return m_new == -INFINITY ? 1.f : (float)exp((double)__fsub_rn(m_old, m_new));
}
// exp(s - m); m = -inf: no score above -inf yet, every term is zero
__device__ __forceinline__ float attn_prob(float s, float m) {
    return (float)exp((double)__fsub_rn(s, m == -INFINITY ? 0.f : m));
}

// The same attention for a run of new tokens (prefill): one block per (kv head, tile of query
// tokens) serves every query head of that kv head -- up to ROWS (token, head) rows -- against
// blocks of kTileKeys keys, with a running softmax (attention_plain_kernel's arithmetic,
// operation for operation: the same bits).  Nothing in the kernel grows with the number of keys.
// What bounds it: the fp32 multiply-adds of the two products (2 * keys * rows * DIM a tile),
// issued two lanes at a time (fma.rn.f32x2); long runs have them on the tensor cores instead
// (attention_tc.cu).  With 64 rows and two blocks per SM one block's softmax (exp in 64 bits) and
// barriers run under the other's products; where there are fewer tiles than that, a tile is a
// serial chain over the keys, which 32 rows shorten.
//   scores   thread = ROWS / 16 rows x 2 keys, 16 bytes of features at a time; shared loads
//            free of bank conflicts (pitch DIM + 4)
//   softmax  256 / ROWS threads per row
//   P*V      thread = ROWS / 16 rows x DIM / 16 features, keys in ascending order
// K of block b + 1 is copied (cp.async) under the softmax and P*V of block b, V of block b
// under its scores; in 4-byte copies where a row is not 16-byte aligned (!ALIGNED; 32 / 8 heads
// of 128, 160 tokens behind 300 keys 93 -> 103 us, one block per (token, head): 730).
// A probability of zero contributes nothing (whatever the value row holds): where an output is
// not finite -- a value row that is not, or values near the largest number added up before the
// division -- the tile runs again with the rows' final maxima and sums, probabilities of zero
// skipped, as attention_kernel has it.
// Measured, 32 / 8 heads of 128, against the former tile kernel (all scores in shared memory,
// one block per (token, head) beyond 1400 keys): 256 tokens 80 -> 39 us, behind 300 keys 131 ->
// 108; 1200 tokens 753 -> 387; 600 tokens behind 1000 keys 3339 -> 512.
template <int DIM, int ROWS>
struct TileSmem {  // floats
    static constexpr int kPitch = DIM + 4, kProbPitch = kTileKeys + 4;
    static constexpr int kQ = 0;
    static constexpr int kK = kQ + ROWS * kPitch;
    static constexpr int kV = kK + kTileKeys * kPitch;
    static constexpr int kP = kV + kTileKeys * kPitch;
    static constexpr int kAlpha = kP + ROWS * kProbPitch;
    static constexpr int kSum = kAlpha + ROWS;
    static constexpr int kBytes = (kSum + ROWS) * 4;
};
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(valid ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Who runs a tile: the whole block, or kAttnThreads threads of a larger one.
struct BlockSync {
    static __device__ __forceinline__ void sync() { __syncthreads(); }
    static __device__ __forceinline__ bool any(bool v) { return __syncthreads_or(v); }
};

// Rows [t0, t0 + tq) of kv head kvh; `tokens` ends the run, `past` keys lie before it.
template <int DIM, int ROWS, bool ALIGNED, typename Sync>
__device__ __forceinline__ void
attention_tile(const float* __restrict__ q, const float* __restrict__ k_cache,
               const float* __restrict__ v_cache, float* __restrict__ out, int tokens, int heads,
               int kv_heads, int past, int capacity, float scale, int tq, int kvh, int t0,
               float* s_dyn) {
    using S = TileSmem<DIM, ROWS>;
    constexpr int RS = kAttnThreads / 16, RT = ROWS / RS;           // rows of a thread, RS apart
    constexpr int ST = kAttnThreads / ROWS, SK = kTileKeys / ST;    // softmax: threads and keys a row
    constexpr int P = S::kPitch, PP = S::kProbPitch;
    float* s_q = s_dyn + S::kQ;
    float* s_k = s_dyn + S::kK;
    float* s_v = s_dyn + S::kV;
    float* s_p = s_dyn + S::kP;
    float* s_alpha = s_dyn + S::kAlpha;
    float* s_sum = s_dyn + S::kSum;
    const int rep = heads / kv_heads;
    const int vis_max = past + min(t0 + tq, tokens);  // keys the tile's last token sees
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
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
    constexpr int kRow4 = DIM / 4;                            // float4 per row
    constexpr int kCopies = kTileKeys * kRow4 / kAttnThreads;  // per thread and block of keys
    auto copy4 = [&](float* dst, const float* src, bool valid) {
        if constexpr (ALIGNED) {
            cp_async16(dst, src, valid);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
                cp_async4(dst + i, src + i, valid);
        }
    };
    auto copy_keys = [&](float* dst, const float* base, int j0) {
#pragma unroll
        for (int u = 0; u < kCopies; ++u) {
            const int i = threadIdx.x + kAttnThreads * u, key = i / kRow4, c = i % kRow4;
            const bool valid = j0 + key < vis_max;
            copy4(dst + key * P + 4 * c, base + (size_t)(valid ? j0 + key : 0) * DIM + 4 * c, valid);
        }
        cp_async_commit();
    };
    for (int i = threadIdx.x; i < ROWS * kRow4; i += kAttnThreads) {
        const int row = i / kRow4, c = i % kRow4;
        const bool live = row_visible(row) > 0;
        copy4(s_q + row * P + 4 * c, q + (live ? row_offset(row) : 0) + 4 * c, live);
    }

    // products: rows ra + RS i, keys kb + 16 j, features 4 kb + 64 i .. + 3
    const int ra = (warp >> 1) * 4 + (lane >> 3), kb = (warp & 1) * 8 + (lane & 7);
    // softmax: row sr, keys SK sq .. SK sq + SK - 1 of a block
    const int sr = threadIdx.x / ST, sq = threadIdx.x % ST;
    const int s_vis = row_visible(sr);
    float m = -INFINITY, l = 0.f;
    bool final_pass = false;  // m and 1 / l are the row's final ones, in m and l
    constexpr int NV = DIM / 64;
    for (;;) {
    copy_keys(s_k, kc, 0);  // the first time with Q: one group
    uint64_t acc[RT][2 * NV];
#pragma unroll
    for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int c = 0; c < 2 * NV; ++c)
            acc[i][c] = 0;

    for (int j0 = 0; j0 < vis_max; j0 += kTileKeys) {
        copy_keys(s_v, vc, j0);
        cp_async_wait<1>();
        Sync::sync();  // K of this block is in place
        {
            float sc[RT][2];
#pragma unroll
            for (int i = 0; i < RT; ++i)
                sc[i][0] = sc[i][1] = 0.f;
#pragma unroll 1
            for (int c = 0; c < DIM; c += 32) {
                uint64_t a[RT][2];
#pragma unroll
                for (int i = 0; i < RT; ++i)
                    a[i][0] = a[i][1] = 0;
#pragma unroll
                for (int d = 0; d < 32; d += 4) {
                    ulonglong2 qv[RT], kv[2];
#pragma unroll
                    for (int i = 0; i < RT; ++i)
                        qv[i] = *reinterpret_cast<const ulonglong2*>(s_q + (ra + RS * i) * P + c + d);
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        kv[j] = *reinterpret_cast<const ulonglong2*>(s_k + (kb + 16 * j) * P + c + d);
#pragma unroll
                    for (int i = 0; i < RT; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j)
                            a[i][j] = b2w4_fma2(qv[i].x, kv[j].x, a[i][j]);
#pragma unroll
                    for (int i = 0; i < RT; ++i)
#pragma unroll
                        for (int j = 0; j < 2; ++j)
                            a[i][j] = b2w4_fma2(qv[i].y, kv[j].y, a[i][j]);
                }
#pragma unroll
                for (int i = 0; i < RT; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        float lo, hi;
                        b2w4_unpack2(a[i][j], lo, hi);
                        sc[i][j] = __fadd_rn(sc[i][j], __fadd_rn(lo, hi));
                    }
            }
#pragma unroll
            for (int i = 0; i < RT; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    s_p[(ra + RS * i) * PP + kb + 16 * j] = __fmul_rn(sc[i][j], scale);
        }
        Sync::sync();  // scores in place, K consumed
        if (j0 + kTileKeys < vis_max)
            copy_keys(s_k, kc, j0 + kTileKeys);
        else
            cp_async_commit();  // an empty group keeps the count
        {
            float* row = s_p + sr * PP + SK * sq;
            float e[SK];
#pragma unroll
            for (int i = 0; i < SK; i += 4)
                *reinterpret_cast<float4*>(e + i) = *reinterpret_cast<const float4*>(row + i);
            float mb = m;
#pragma unroll
            for (int i = 0; i < SK; ++i)
                if (j0 + SK * sq + i < s_vis)
                    mb = fmaxf(mb, e[i]);
#pragma unroll
            for (int off = 1; off < ST; off <<= 1)
                mb = fmaxf(mb, __shfl_xor_sync(0xffffffffu, mb, off));
            const float alpha = j0 && !final_pass ? attn_rescale(m, mb) : 1.f;
            m = mb;  // final_pass: as it was
#pragma unroll
            for (int i = 0; i < SK; ++i)
                e[i] = j0 + SK * sq + i < s_vis ? attn_prob(e[i], m) : 0.f;
            if (final_pass) {
#pragma unroll
                for (int i = 0; i < SK; ++i)
                    e[i] = __fmul_rn(e[i], l);
            }
#pragma unroll
            for (int i = 0; i < SK; i += 4)
                *reinterpret_cast<float4*>(row + i) = *reinterpret_cast<const float4*>(e + i);
#pragma unroll
            for (int n = 1; n < SK; n <<= 1)
#pragma unroll
                for (int i = 0; i < SK; i += 2 * n)
                    e[i] = __fadd_rn(e[i], e[i + n]);
            float sum = e[0];
#pragma unroll
            for (int off = 1; off < ST; off <<= 1)
                sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, off));
            if (!final_pass)
                l = __fadd_rn(__fmul_rn(l, alpha), sum);
            if (sq == 0)
                s_alpha[sr] = alpha;
        }
        cp_async_wait<1>();  // V of this block
        Sync::sync();  // V, probabilities, factors in place
#pragma unroll
        for (int i = 0; i < RT; ++i) {
            const float al = s_alpha[ra + 16 * i];
            if (al != 1.f) {
                const uint64_t al2 = b2w4_pack2(al, al);
#pragma unroll
                for (int c = 0; c < 2 * NV; ++c)
                    acc[i][c] = al == 0.f ? 0 : b2w4_mul2(acc[i][c], al2);
            }
        }
        if (!final_pass) {
#pragma unroll 2
            for (int j = 0; j < kTileKeys; j += 4) {
                float4 p4[RT];
#pragma unroll
                for (int i = 0; i < RT; ++i)
                    p4[i] = *reinterpret_cast<const float4*>(s_p + (ra + RS * i) * PP + j);
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    ulonglong2 v[NV];
#pragma unroll
                    for (int c = 0; c < NV; ++c)
                        v[c] = *reinterpret_cast<const ulonglong2*>(s_v + (j + jj) * P + 4 * kb +
                                                                    64 * c);
#pragma unroll
                    for (int i = 0; i < RT; ++i) {
                        const float p = jj == 0 ? p4[i].x : jj == 1 ? p4[i].y
                                      : jj == 2 ? p4[i].z : p4[i].w;
                        const uint64_t pp = b2w4_pack2(p, p);
#pragma unroll
                        for (int c = 0; c < NV; ++c) {
                            acc[i][2 * c] = b2w4_fma2(v[c].x, pp, acc[i][2 * c]);
                            acc[i][2 * c + 1] = b2w4_fma2(v[c].y, pp, acc[i][2 * c + 1]);
                        }
                    }
                }
            }
        } else {
#pragma unroll 1
            for (int j = 0; j < kTileKeys; ++j) {
#pragma unroll
                for (int i = 0; i < RT; ++i) {
                    const float p = s_p[(ra + RS * i) * PP + j];
                    if (p != 0.f) {
                        const uint64_t pp = b2w4_pack2(p, p);
#pragma unroll
                        for (int c = 0; c < NV; ++c) {
                            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(
                                s_v + j * P + 4 * kb + 64 * c);
                            acc[i][2 * c] = b2w4_fma2(v.x, pp, acc[i][2 * c]);
                            acc[i][2 * c + 1] = b2w4_fma2(v.y, pp, acc[i][2 * c + 1]);
                        }
                    }
                }
            }
        }
        Sync::sync();  // V and the probabilities are consumed
    }
    if (sq == 0)
        s_sum[sr] = final_pass ? 1.f : l;
    Sync::sync();
    bool odd = false;
#pragma unroll
    for (int i = 0; i < RT; ++i) {
        const int row = ra + RS * i;
        if (row_visible(row)) {
            const float total = s_sum[row];
#pragma unroll
            for (int c = 0; c < NV; ++c) {
                float4 o;
                b2w4_unpack2(acc[i][2 * c], o.x, o.y);
                b2w4_unpack2(acc[i][2 * c + 1], o.z, o.w);
                o.x = __fdiv_rn(o.x, total);
                o.y = __fdiv_rn(o.y, total);
                o.z = __fdiv_rn(o.z, total);
                o.w = __fdiv_rn(o.w, total);
                // inf and NaN, times zero, are NaN
                const float z = __fadd_rn(__fadd_rn(__fmul_rn(o.x, 0.f), __fmul_rn(o.y, 0.f)),
                                          __fadd_rn(__fmul_rn(o.z, 0.f), __fmul_rn(o.w, 0.f)));
                odd |= z != 0.f;
                float* dst = out + row_offset(row) + 4 * kb + 64 * c;
                if constexpr (ALIGNED) {
                    *reinterpret_cast<float4*>(dst) = o;
                } else {
                    dst[0] = o.x;
                    dst[1] = o.y;
                    dst[2] = o.z;
                    dst[3] = o.w;
                }
            }
        }
    }
    cp_async_wait<0>();
    if (final_pass || !Sync::any(odd))
        return;
    final_pass = true;
    l = __fdiv_rn(1.f, l);
    }
}

}  // namespace
