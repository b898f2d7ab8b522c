// k_gemm_tc.cuh -- device pieces of the tcgen05 products: shared-memory and instruction
// descriptors, the bounded mbarrier wait, and the no-swizzle K-major tile layout.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "fwt_internal.h"

namespace fwt {

constexpr int kGemmBM = 128, kGemmBK = 64;

__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    // start address, leading and stride byte offsets in 16-byte units; bits 46-47 = 1 (the
    // sm_100 descriptor version); layout type 0 (no swizzle) in bits 61-63, base offset 0
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ uint32_t umma_idesc_bf16(int M, int N)
{
    // D F32 (bits 4-5 = 1), A BF16 (bits 7-9 = 1), B BF16 (bits 10-12 = 1), both K-major,
    // N >> 3 in bits 17-22, M >> 4 in bits 24-28
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ bool gemm_mbar_wait(uint32_t bar, uint32_t phase)
{
    for (int it = 0; it < (1 << 24); ++it) {
        uint32_t done;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// byte offset of element (row r, k) of a rows x 64 K-major no-swizzle tile
__device__ __forceinline__ uint32_t core_off(int r, int k8, int rows)
{
    return (uint32_t)(k8 * rows * 16 + (r >> 3) * 128 + (r & 7) * 16);
}

}  // namespace fwt
