// Small wrappers of the tcgen05 / mbarrier instructions that the tensor-core kernels share.
#pragma once
#include <cstdint>

namespace shm {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

constexpr int kSpinLimit = 1 << 24;  // polls of a wait on an mbarrier (1.5 us each when nothing comes)

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int limit = kSpinLimit) {
    for (int it = 0; it < limit; it++)
        if (mbar_try(bar, parity)) return true;
    return false;
}

// K-major, no-swizzle ("interleaved") operand with rows of 64 bytes: core matrices of 8 rows x 16
// bytes, K-adjacent core matrices 128 B apart (LBO), 8-row groups 512 B apart (SBO).
constexpr uint32_t kKB = 64;
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)(128 >> 4) << 16;             // leading byte offset (K direction)
    d |= (uint64_t)((kKB / 16 * 128) >> 4) << 32;  // stride byte offset (M/N direction)
    d |= (uint64_t)1 << 46;                      // descriptor version for sm_100
    return d;                                    // base offset 0, lbo mode 0, layout SWIZZLE_NONE
}

// byte offset of (row, 16-byte chunk kc) inside an operand of rows of kKB bytes
__device__ __forceinline__ uint32_t core_off(uint32_t row, uint32_t kc) {
    return ((row >> 3) * (kKB / 16) + kc) * 128 + (row & 7) * 16;
}

}  // namespace shm
