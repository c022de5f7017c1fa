// What the tensor-core kernels share: descriptors of tcgen05.mma and the bounded wait of their roles.
#pragma once

#include "coll_common.cuh"

namespace yali {

// Shared-memory matrix descriptor of a K-major operand tile stored by TMA with 128-byte
// swizzle: rows of 128 bytes, groups of 8 rows 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((smem_addr & 0x3ffffu) >> 4);  // start address
    d |= static_cast<uint64_t>(1) << 16;                      // leading byte offset (unused with swizzle)
    d |= static_cast<uint64_t>(1024 >> 4) << 32;              // stride byte offset: next 8-row group
    d |= static_cast<uint64_t>(1) << 46;                      // descriptor version of sm_100
    d |= static_cast<uint64_t>(2) << 61;                      // SWIZZLE_128B
    return d;
}

// Instruction descriptor: D = fp32, A = B = bf16, both K-major, N at bit 17 (>>3), M at bit 24 (>>4).
__device__ __forceinline__ uint32_t mma_idesc_bf16(uint32_t m, uint32_t n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// Wait of a role of a pair of CTAs: gives up at the deadline or when another role of this CTA has.
__device__ __forceinline__ bool wait_bar(uint64_t* bar, uint32_t parity, uint64_t deadline, volatile int* abort) {
    uint32_t tries = 0;
    while (!ptx::mbar_try_wait_cluster(bar, parity)) {
        if ((++tries & 15u) == 0 && (*abort || ptx::globaltimer() > deadline)) return false;
    }
    return true;
}

}  // namespace yali
