// W4G128 x int8 matmul for a few activation rows (9..32, and 2..8 by few_rows_streamed in capi.cu:
// batched decode, short prompts) on the warp-level int8 tensor instruction (mma.sync m16n8k32).
//
// Arithmetic = the reference's, row by row, under either rule (kernels/matmul_w4.cpp:211-295 with
// one activation scale per 128 values, :785-901 with one per 32): per group or 32-k block
//   D = sum q4*q8 (int32);  y = fma(float(D), fp32(ws*as), y)
// in ascending order.  The chain value of every (row, weight row) stays in one register of one
// thread for the whole K loop.
//
// Work split.  A warp owns a pair of 8-row weight tiles (the sixteen rows of the instruction) and
// all blocks of eight activation rows (its columns), or, where there are few pairs, several warps
// share a pair; a CTA holds up to ten warps (sixteen where pairs are shared), so that one or two
// CTAs per SM take a weight of up to twenty pairs per SM in one round.  Weights, codes and scales stream through a ring of shared-memory stages of four
// groups, one barrier per stage; the weights of the first stages are on their way before the
// kernel waits for the quantiser in front (programmatic dependent launch).  (Fetched into
// registers four groups ahead instead, the weights came no sooner: a warp's outstanding loads
// share six scoreboards, so a wait for an old group waited for the newest too; 16 rows,
// [9728, 2560], 23.5 us.)
// A weight word is split into signed bytes 16 q (lo = (w << 4) & 0xF0F0F0F0: even k; hi = w &
// 0xF0F0F0F0: odd k).  Every accumulator starts at 0x49400000, the bits of the float 786432 whose
// last place is worth 1/16, and ends as the bits of 786432 + D, exactly, since
// |16 D| <= 128 * 127 * 128 < 2^22: D costs one subtraction, for two columns at once.  (Unsigned
// bytes q + 8 need a start that depends on the sum of the codes, four more words per instruction
// to make, copy and read: 16 rows, [9728, 2560], per 32 values, 11.1 -> 9.6 us.)
//
// What bounds it: the latency of few warps.  16 rows of [9728, 2560] per 32 values, ten warps per
// SM: issue slots 45 % busy, DRAM 13 %, a warp waits 5.4 cycles per instruction (1.5 for the result
// before it, 0.6 for the fp32 pipe, 0.5 at the stage's barrier).
#include "b200w4_internal.cuh"

namespace {

constexpr int kRowsWarps = 10;        // warps per CTA at most
constexpr int kRowsThreads = kRowsWarps * 32;
constexpr int kChunk = 4;             // groups per stage
constexpr int kRelayWarps = 16;       // the same where warps share a chain
constexpr int kPitch = kChunk * 128 + 16;  // bytes between a stage's rows: conflict-free reads

struct GemmRowsArgs {
    const uint8_t* nib;
    const void* scl;
    const int8_t* qa;    // [m][K] int8, tensor-operand order inside each group
    const float* as_t;   // activation scales [G][m8], per 32 values [G][m8 / 2][4 blocks][2 rows]
    float* y;
    int ldc, m, m8, n, k, groups, tiles, pairs;
    int pw;              // KS > 1: warps beside one another per pair, one column block each
    int activation, act_n_begin, act_n_len;
};

__device__ __forceinline__ void rows_cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
// lane (gid = lane/4, tid = lane%4): a0 row gid, k 4*tid..+3; a1 row gid+8; a2/a3 k+16;
// b0 k 4*tid..+3 of column gid, b1 k+16; d0/d1 row gid, columns 2*tid, 2*tid+1; d2/d3 row gid+8
__device__ __forceinline__ void rows_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1, int4 c) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%10,%11,%12,%13};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c.x), "r"(c.y), "r"(c.z),
          "r"(c.w));
}

__device__ __noinline__ float rows_activation(float v, int act) { return b2w4_activation(v, act); }

__host__ __device__ constexpr size_t rows_stage_bytes(int m8, int spg, int pairs, bool scl16) {
    return (size_t)m8 * (kPitch + kChunk * spg * 4) +
           (size_t)pairs * 2 * kChunk * (512 + (scl16 ? 16 : 32));
}

// PW warps per pair of weight tiles, CB blocks of eight activation rows per warp, S stages.
// KS > 1 (few pairs): KS warps share a pair and a column block (PW is not used, a.pw is).  Each
// takes kChunk / KS groups of a stage, makes their sums and products ws * as, and only then
// needs the chain values: it has them from the warp that holds the groups before, through shared
// memory, and hands them on, so that the chain keeps its order.
template <int PW, int CB, bool SCL16, bool A32, int S, int KS>
__global__ void __launch_bounds__(KS > 1 ? kRelayWarps * 32 : kRowsThreads, KS > 1 ? 1 : 2)
gemm_w4a8_rows_kernel(const GemmRowsArgs a) {
    constexpr int SPG = A32 ? 4 : 1;  // scales per group
    constexpr int kScl = SCL16 ? 16 : 32;  // bytes of a tile's scales of a group
    extern __shared__ __align__(128) uint8_t smem[];
    const int G = a.groups, m8 = a.m8;
    const int pw = KS > 1 ? a.pw : PW;
    const int warps = blockDim.x / 32, pairs = warps / (pw * KS);
    const int as_bytes = kChunk * SPG * m8 * 4;
    const int nib_off = as_bytes + m8 * kPitch;
    const int scl_off = nib_off + pairs * 2 * kChunk * 512;
    const int stage_bytes = (int)rows_stage_bytes(m8, SPG, pairs, SCL16);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tid = lane & 3;
    const int chain = warp / KS, turn = warp % KS;
    const int pair0 = blockIdx.x * pairs, pair = pair0 + chain / pw;
    const int cb0 = (chain % pw) * CB;  // first column block
    const int ncb = PW == 1 || KS > 1 ? CB : min(CB, m8 / 8 - cb0);  // may be none
    const bool busy = pair < a.pairs && ncb > 0;
    const int t0 = 2 * pair;
    const bool two = t0 + 1 < a.tiles;
    const int tiles_here = min(2 * pairs, a.tiles - 2 * pair0);
    const int chunks = (G + kChunk - 1) / kChunk;

    b2w4_pdl_launch_dependents();
    // stage: [tile][group of the chunk][512], then [tile][group][8 scales]
    auto load_weights = [&](int c) {
        if (c < chunks) {
            uint8_t* s = smem + (c % S) * stage_bytes;
            const int g0 = c * kChunk, gc = min(kChunk, G - g0);
            const int n16 = gc * 32, s16 = gc * (kScl / 16);
            for (int t = warp; t < tiles_here; t += warps) {  // a tile per warp
                const size_t at = (size_t)(2 * pair0 + t) * G + g0;
                for (int i = lane; i < n16; i += 32)
                    rows_cp_async16(s + nib_off + t * (kChunk * 512) + i * 16,
                                    a.nib + at * 512 + i * 16);
                if (lane < s16)
                    rows_cp_async16(s + scl_off + t * (kChunk * kScl) + lane * 16,
                                    reinterpret_cast<const uint8_t*>(a.scl) + at * kScl + lane * 16);
            }
        }
    };
#pragma unroll
    for (int c = 0; c < S - 1; ++c)
        load_weights(c);

    b2w4_pdl_wait();  // quantised activations come from the previous kernel
    auto load_rows = [&](int c) {
        if (c < chunks) {
            uint8_t* s = smem + (c % S) * stage_bytes;
            const int g0 = c * kChunk, gc = min(kChunk, G - g0);
            const int n_as = gc * SPG * m8 / 4, n_row = gc * 8;
            const float* as = a.as_t + (size_t)g0 * SPG * m8;
            for (int i = threadIdx.x; i < n_as; i += blockDim.x)
                rows_cp_async16(s + i * 16, as + i * 4);
            uint8_t* rows = s + as_bytes;
            for (int t = warp; t < a.m; t += warps)
                if (lane < n_row)
                    rows_cp_async16(rows + t * kPitch + lane * 16,
                                    a.qa + (size_t)t * a.k + (size_t)g0 * 128 + lane * 16);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int c = 0; c < S - 1; ++c)
        load_rows(c);

    uint64_t acc[CB][2];  // [0]: row gid, columns 2*tid and 2*tid+1; [1]: row gid+8
#pragma unroll
    for (int j = 0; j < CB; ++j)
        acc[j][0] = acc[j][1] = 0ull;
    const uint64_t magic = b2w4_pack2(786432.f, 786432.f);
    const int4 start = make_int4(0x49400000, 0x49400000, 0x49400000, 0x49400000);

#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncthreads();  // stage c visible to all; everyone is done with stage c-1
        load_weights(c + S - 1);
        load_rows(c + S - 1);
        const uint8_t* s = smem + (c % S) * stage_bytes;
        // the scales of row pair 4 * cb0 + tid of the first group
        const uint64_t* s_as = reinterpret_cast<const uint64_t*>(s) + (cb0 * 4 + tid) * SPG;
        const uint8_t* rows = s + as_bytes + (cb0 * 8 + gid) * kPitch + tid * 32;
        // this lane's words: row gid of each tile, bytes 4*tid..+3 of every 32-k block
        const int tl = t0 - 2 * pair0;
        const uint32_t* s_w = reinterpret_cast<const uint32_t*>(s + nib_off) + tl * (kChunk * 128) + lane;
        const uint8_t* s_scl = s + scl_off + tl * (kChunk * kScl) + gid * (kScl / 8);
        // the words of group i of the stage, split, and the scales of both tiles
        auto words = [&](int i, uint32_t (&lo)[2][4], uint32_t (&hi)[2][4], uint64_t (&ws2)[2]) {
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const bool have = t == 0 || two;  // a missing tile: zeros
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const uint32_t w = have ? s_w[t * (kChunk * 128) + i * 128 + b * 32] : 0u;
                    lo[t][b] = (w << 4) & 0xF0F0F0F0u;
                    hi[t][b] = w & 0xF0F0F0F0u;
                }
                const uint8_t* q = s_scl + t * (kChunk * kScl) + i * kScl;
                const float ws = !have  ? 0.f
                                 : SCL16 ? __half2float(*reinterpret_cast<const __half*>(q))
                                         : *reinterpret_cast<const float*>(q);
                ws2[t] = b2w4_pack2(ws, ws);
            }
        };
        // the sums of a group, per block (A32) or whole, of column block j
        auto sums = [&](int i, int j, const uint32_t (&lo)[2][4], const uint32_t (&hi)[2][4],
                        int (&d)[SPG][4]) {
            const uint4* bp = reinterpret_cast<const uint4*>(rows + j * 8 * kPitch + i * 128);
            const uint4 be = bp[0], bo = bp[1];
            const uint32_t bev[4] = {be.x, be.y, be.z, be.w};
            const uint32_t bov[4] = {bo.x, bo.y, bo.z, bo.w};
            if (A32) {
#pragma unroll
                for (int b = 0; b < SPG; ++b)  // one instruction = one 32-block
                    rows_mma(d[b], lo[0][b], lo[1][b], hi[0][b], hi[1][b], bev[b], bov[b], start);
            } else {
                // two chains of two instructions (latency), joined by one add
                int e[4];
                rows_mma(d[0], lo[0][0], lo[1][0], hi[0][0], hi[1][0], bev[0], bov[0], start);
                rows_mma(e, lo[0][1], lo[1][1], hi[0][1], hi[1][1], bev[1], bov[1],
                         make_int4(0, 0, 0, 0));
                rows_mma(d[0], lo[0][2], lo[1][2], hi[0][2], hi[1][2], bev[2], bov[2],
                         make_int4(d[0][0], d[0][1], d[0][2], d[0][3]));
                rows_mma(e, lo[0][3], lo[1][3], hi[0][3], hi[1][3], bev[3], bov[3],
                         make_int4(e[0], e[1], e[2], e[3]));
#pragma unroll
                for (int x = 0; x < 4; ++x)
                    d[0][x] += e[x];
            }
        };
        auto scales = [&](int i, int j, uint64_t (&as2)[SPG]) {
            const uint64_t* at = s_as + (i * (m8 / 2) + j * 4) * SPG;
            if (A32) {
                const ulonglong2 a01 = reinterpret_cast<const ulonglong2*>(at)[0];
                const ulonglong2 a23 = reinterpret_cast<const ulonglong2*>(at)[1];
                as2[0] = a01.x, as2[SPG / 4] = a01.y, as2[SPG / 2] = a23.x, as2[SPG - 1] = a23.y;
            } else {
                as2[0] = at[0];
            }
        };
        // d = 0x49400000 + 16 D: as a float 786432 + D, exactly
        auto value = [&](int x, int y) {
            return b2w4_sub2(b2w4_pack2(__int_as_float(x), __int_as_float(y)), magic);
        };
        if constexpr (KS > 1) {
            constexpr int GPW = kChunk / KS;
            uint64_t v[GPW][SPG][2], f[GPW][SPG][2];
#pragma unroll
            for (int i = 0; i < GPW; ++i) {
                const int at = turn * GPW + i;
                if (c * kChunk + at < G && busy) {  // warp-uniform
                    uint32_t lo[2][4], hi[2][4];
                    uint64_t ws2[2], as2[SPG];
                    int d[SPG][4];
                    words(at, lo, hi, ws2);
                    scales(at, 0, as2);
                    sums(at, 0, lo, hi, d);
#pragma unroll
                    for (int b = 0; b < SPG; ++b) {
                        v[i][b][0] = value(d[b][0], d[b][1]);
                        v[i][b][1] = value(d[b][2], d[b][3]);
                        f[i][b][0] = b2w4_mul2(ws2[0], as2[b]);
                        f[i][b][1] = b2w4_mul2(ws2[1], as2[b]);
                    }
                }
            }
            // The chain values: from the warp in front (the first one's come from the last one,
            // before the barrier of this stage).  Barriers 1..12: (KS - 1) links of each chain.
            ulonglong2* s_y =
                reinterpret_cast<ulonglong2*>(smem + S * stage_bytes) + chain * 32 + lane;
            const int link = 1 + chain * (KS - 1) + turn;
            if (turn > 0)
                asm volatile("bar.sync %0, 64;" ::"r"(link - 1) : "memory");
            if (c > 0 || turn > 0) {
                const ulonglong2 y2 = *s_y;
                acc[0][0] = y2.x;
                acc[0][1] = y2.y;
            }
#pragma unroll
            for (int i = 0; i < GPW; ++i)
                if (c * kChunk + turn * GPW + i < G && busy) {
#pragma unroll
                    for (int b = 0; b < SPG; ++b) {
                        acc[0][0] = b2w4_fma2(v[i][b][0], f[i][b][0], acc[0][0]);
                        acc[0][1] = b2w4_fma2(v[i][b][1], f[i][b][1], acc[0][1]);
                    }
                }
            *s_y = make_ulonglong2(acc[0][0], acc[0][1]);
            if (turn < KS - 1)
                asm volatile("bar.arrive %0, 64;" ::"r"(link) : "memory");
            continue;
        }
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
            if (c * kChunk + i < G && busy) {  // warp-uniform
                uint32_t lo[2][4], hi[2][4];
                uint64_t ws2[2];
                words(i, lo, hi, ws2);
#pragma unroll
                for (int j = 0; j < CB; ++j) {
                    if (j < ncb) {
                        uint64_t as2[SPG];
                        int d[SPG][4];
                        scales(i, j, as2);
                        sums(i, j, lo, hi, d);
#pragma unroll
                        for (int b = 0; b < SPG; ++b) {  // blocks in ascending order
                            acc[j][0] = b2w4_fma2(value(d[b][0], d[b][1]),
                                                  b2w4_mul2(ws2[0], as2[b]), acc[j][0]);
                            acc[j][1] = b2w4_fma2(value(d[b][2], d[b][3]),
                                                  b2w4_mul2(ws2[1], as2[b]), acc[j][1]);
                        }
                    }
                }
            }
        }
    }

    // y[row][n]: for one row, the eight lanes of a quarter-warp hold eight consecutive n
    if (busy && turn == KS - 1) {
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const int n = (t0 + t) * 8 + gid;
            const bool act = b2w4_act_applies(n, a.activation, a.act_n_begin, a.act_n_len, a.n);
#pragma unroll
            for (int j = 0; j < CB; ++j) {
                float v[2];
                b2w4_unpack2(acc[j][t], v[0], v[1]);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    const int r = (cb0 + j) * 8 + tid * 2 + x;
                    if (r < a.m && n < a.n)
                        a.y[(size_t)r * a.ldc + n] = act ? rows_activation(v[x], a.activation) : v[x];
                }
            }
        }
    }
}

template <int PW, int CB, bool SCL16, bool A32, int S, int KS>
int rows_launch_as(b2w4_ctx* ctx, const GemmRowsArgs& a, int pairs_per_cta) {
    auto kern = gemm_w4a8_rows_kernel<PW, CB, SCL16, A32, S, KS>;
    const int chains = pairs_per_cta * (KS > 1 ? a.pw : PW);
    const size_t smem = S * rows_stage_bytes(a.m8, A32 ? 4 : 1, pairs_per_cta, SCL16) +
                        (KS > 1 ? chains * 512 : 0);
    static b2w4_smem_optin configured;  // per instantiation and device
    B2W4_CUDA(ctx, b2w4_opt_in_smem(ctx, kern, smem, configured));
    B2W4_CUDA(ctx, b2w4_launch_chained(ctx->pdl, kern,
                                       dim3((a.pairs + pairs_per_cta - 1) / pairs_per_cta),
                                       dim3(chains * KS * 32), smem, ctx->stream, a));
    ctx->launches++;
    return B2W4_OK;
}
// whether a CTA has the SM to itself and room for so many stages
bool rows_deep(b2w4_ctx* ctx, const GemmRowsArgs& a, bool scl16, bool a32, int pairs_per_cta,
               int stages) {
    return (a.pairs + pairs_per_cta - 1) / pairs_per_cta <= ctx->sm_count &&
           stages * rows_stage_bytes(a.m8, a32 ? 4 : 1, pairs_per_cta, scl16) <= 220 * 1024;
}
template <int PW, int CB, bool SCL16, bool A32>
int rows_launch(b2w4_ctx* ctx, const GemmRowsArgs& a, int pairs_per_cta) {
    // six stages, or five where six do not fit (32 rows of [9728, 2560] per 128 values: three
    // stages 16.7 us, five 11.9), else three for two CTAs
    if (rows_deep(ctx, a, SCL16, A32, pairs_per_cta, 6))
        return rows_launch_as<PW, CB, SCL16, A32, 6, 1>(ctx, a, pairs_per_cta);
    return rows_deep(ctx, a, SCL16, A32, pairs_per_cta, 5)
               ? rows_launch_as<PW, CB, SCL16, A32, 5, 1>(ctx, a, pairs_per_cta)
               : rows_launch_as<PW, CB, SCL16, A32, 3, 1>(ctx, a, pairs_per_cta);
}
template <bool SCL16, bool A32>
int rows_relay(b2w4_ctx* ctx, const GemmRowsArgs& a, int pairs_per_cta) {
    return pairs_per_cta * a.pw * 4 <= kRelayWarps
               ? rows_launch_as<1, 1, SCL16, A32, 6, 4>(ctx, a, pairs_per_cta)
               : rows_launch_as<1, 1, SCL16, A32, 6, 2>(ctx, a, pairs_per_cta);
}

}  // namespace

size_t b2w4_rows_scratch(const b2w4_weight* w, int m, int act_rule) {
    const int spg = act_rule == B2W4_ACT_G32 ? 4 : 1, m8 = (m + 7) & ~7;
    return (size_t)m * w->k + sizeof(float) * w->groups * spg * m8;
}

int b2w4_launch_gemm_rows(b2w4_ctx* ctx, const b2w4_weight* w, const float* x, int lda, float* y,
                          int ldc, int m, int act_rule, int activation, int act_n_begin,
                          int act_n_len, const b2w4_rows* from, void* own) {
    const bool a32 = act_rule == B2W4_ACT_G32;
    const int G = w->groups, spg = a32 ? 4 : 1, m8 = (m + 7) & ~7;
    void *qa = own, *sc = nullptr;
    int rc;
    if (own)  // k is whole groups of 128: the scales stay aligned
        sc = static_cast<uint8_t*>(own) + (size_t)m * w->k;
    else if ((rc = b2w4_reserve(ctx, SCR_QA, (size_t)m * w->k, &qa)) != B2W4_OK ||
             (rc = b2w4_reserve(ctx, SCR_AS, sizeof(float) * G * spg * m8, &sc)) != B2W4_OK)
        return rc;
    float* as_t = static_cast<float*>(sc);
    if ((rc = b2w4_launch_quantize_rows(ctx, x, lda, m, w->k, m8, act_rule,
                                        static_cast<int8_t*>(qa), as_t, from)) != B2W4_OK)
        return rc;
    GemmRowsArgs a;
    a.nib = reinterpret_cast<const uint8_t*>(w->nib);
    a.scl = w->scl;
    a.qa = static_cast<const int8_t*>(qa);
    a.as_t = as_t;
    a.y = y;
    a.ldc = ldc;
    a.m = m;
    a.m8 = m8;
    a.n = w->n;
    a.k = w->k;
    a.groups = G;
    a.tiles = w->tiles;
    a.pairs = (w->tiles + 1) / 2;
    a.activation = activation;
    a.act_n_begin = act_n_begin;
    a.act_n_len = act_n_len;
    // Warps per pair: one, which splits a weight word once for all column blocks, while that
    // gives every scheduler a warp; with fewer pairs the column blocks go to several.
    const int ncb = m8 / 8, room = 10 * ctx->sm_count;
    int pw = 1;
    if (ncb == 2 || ncb == 4)
        pw = a.pairs * 2 <= room ? 2 : 1;
    else if (ncb == 3)
        pw = a.pairs * 3 <= room ? 3 : 1;
    const bool scl16 = w->scales_fp16 != 0;
    // Few pairs per SM: a warp's latency sets the time, so two or four warps share a chain.  Per
    // 32 values the chain itself is four times as long: with three pairs per SM or more it is
    // shared for one column block only, and with three or four not at all.  us per call before
    // -> after, per 32 / per 128 values: [2560, 9728]
    // 8 rows 24.2 -> 20.3 / 23.6 -> 18.6, 16 rows 26.0 -> 21.3 / 24.3 -> 19.1, 32 rows 33.0 ->
    // 28.4 / 31.9 -> 23.5; [9728, 2560] (five pairs) 8 rows 8.4 -> 7.7 / 8.0 -> 7.0; [6144, 2560]
    // (three) 8 rows 6.7 -> 7.1, not taken / 6.8 -> 6.3, 16 rows 7.9 -> 8.1, not taken / 7.6 -> 7.2.
    // Other row lengths, pairs per SM x column blocks (those of more than sixteen warps are not
    // shared): K = 4096 per 32 1 x 1 12.4 -> 9.3, 1 x 4 17.3 -> 11.0, 2 x 2 12.2 -> 10.6, 5 x 1
    // 12.5 -> 11.8; per 128 1 x 4 17.1 -> 10.0, 3 x 2 11.0 -> 10.3, 4 x 2 11.3 -> 11.1; K = 1024 from
    // 0.7 less to 0.4 more.  The line is not the best everywhere: per 32 2 x 4 is slower than
    // unshared up to K = 4096 (1024 5.2 -> 6.6, 2560 9.4 -> 10.9, 4096 14.4 -> 15.2; 9728 33.1 ->
    // 29.8), and 7 x 1 is (2560 8.9 -> 11.5, 4096 13.1 -> 15.6).
    a.pw = ncb;
    const int few = (a.pairs + ctx->sm_count - 1) / ctx->sm_count;
    if (few * ncb * 2 <= kRelayWarps && (few <= 2 || !a32 || (few > 4 && ncb == 1)) &&
        rows_deep(ctx, a, scl16, a32, few, 6))
        return scl16 ? (a32 ? rows_relay<true, true>(ctx, a, few)
                            : rows_relay<true, false>(ctx, a, few))
                     : (a32 ? rows_relay<false, true>(ctx, a, few)
                            : rows_relay<false, false>(ctx, a, few));
    // Pairs per CTA: the fullest SM decides, so the least (CTAs on it) x (pairs of each); a CTA's
    // own share of the activations counts as half a pair.
    int best = 1;
    long best_cost = -1;
    for (int p = 1; p <= kRowsWarps / pw; ++p) {
        const long ctas = (a.pairs + p - 1) / p;
        const long cost = (ctas + ctx->sm_count - 1) / ctx->sm_count * (2 * p + 1);
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = p;
        }
    }
#define B2W4_ROWS(PW, CB)                                                                \
    (scl16 ? (a32 ? rows_launch<PW, CB, true, true>(ctx, a, best)                        \
                  : rows_launch<PW, CB, true, false>(ctx, a, best))                      \
           : (a32 ? rows_launch<PW, CB, false, true>(ctx, a, best)                       \
                  : rows_launch<PW, CB, false, false>(ctx, a, best)))
    switch (ncb * 8 + pw) {
    case 1 * 8 + 1: return B2W4_ROWS(1, 1);
    case 2 * 8 + 1: return B2W4_ROWS(1, 2);
    case 2 * 8 + 2: return B2W4_ROWS(2, 1);
    case 3 * 8 + 1: return B2W4_ROWS(1, 3);
    case 3 * 8 + 3: return B2W4_ROWS(3, 1);
    case 4 * 8 + 1: return B2W4_ROWS(1, 4);
    default: return B2W4_ROWS(2, 2);
    }
#undef B2W4_ROWS
}
