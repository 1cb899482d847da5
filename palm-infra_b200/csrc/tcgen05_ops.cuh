// What the tcgen05 kernels share (one translation unit per kernel family): arguments,
// mbarrier, bulk-copy, tensor-core and tensor-memory primitives.
#pragma once

#include "b200w4_internal.cuh"

namespace {

constexpr unsigned kSpinLimit = 1u << 24;
constexpr unsigned long long kWaitLimitCycles = 4000000000ull;  // SM cycles: about 2 s

struct GemmArgs {
    const uint8_t* nib;  // [tiles][G][512]
    const void* scl;     // [tiles][G][8] fp16|fp32
    const int8_t* qa;    // [G][m_pad][128] int8, 16-byte chunks swizzled by token%8
    const float* as;     // [G][m_pad]; per-32 rule: [G][m_pad][4], one scale per 32-k block
    float* y;
    int* status;
    int ldc, m, m_pad, n, groups, tiles;
    int rows_per_cta;  // R
    int activation, act_n_begin, act_n_len;
};

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
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Without a suspend-time hint: with one, waiting threads stay out of the working warps' issue
// slots but wake late (per-32 matmul, [4100, 9728]: 33 rows 43.9 us with a hint of 20 us, 41.1
// without; 1000 rows 209 / 206).
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
// false when the iteration or the time limit runs out
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity))
        return true;
    const unsigned long long t0 = wait_clock();
    for (unsigned spins = 0; spins < kSpinLimit; ++spins) {
        if (mbar_try_wait(bar, parity))
            return true;
        if ((spins & 255) == 255 && wait_clock() - t0 > kWaitLimitCycles)
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

// K-major operand, 128-byte swizzle, 8-row atoms of 1024 bytes packed back to back:
// start address >> 4 in bits [0,14), leading byte offset (unused for swizzled K-major) = 1
// in [16,30), stride byte offset 1024 >> 4 in [32,46), descriptor version 1 in [46,48),
// layout type SWIZZLE_128B = 2 in [61,64).
__device__ __forceinline__ uint64_t umma_desc_k_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// True in one lane (the same one every time) of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(one));
    return one != 0;
}
// kind::i8, int32 accumulate, signed 8-bit A and B, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t umma_idesc_i8(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void umma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "r"(taddr)
        : "memory");
}

__device__ __noinline__ float gemm_activation(float v, int act) {
    return b2w4_activation(v, act);
}

constexpr int kGC = 4;  // groups per raw-weight chunk

}  // namespace
