// Device pieces shared by the tcgen05 kernels: bounded mbarrier waits, TMA loads, K-major
// 128-byte-swizzled operand descriptors.
#pragma once
#include <cuda.h>

#include <cstdint>

namespace hdg {

constexpr long long kSpinLimit = 1ll << 26;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
    for (long long it = 0; it < kSpinLimit; it++) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred P1;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P1;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3fff);
    d |= (uint64_t)1 << 16;                   // leading byte offset (unused by K-major SW128)
    d |= (uint64_t)(1024 >> 4) << 32;         // stride byte offset: 8 rows x 128 bytes
    d |= (uint64_t)1 << 46;                   // descriptor version (sm100)
    d |= (uint64_t)2 << 61;                   // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// Tensor map of a row-major bf16 [n x d] matrix read in boxes of 64 (K) x box_rows, 128-byte
// swizzle, zero fill past the edges (hdg_gemm.cu)
CUtensorMap bf16_rows_map(const void* base, uint64_t n, int d, uint32_t box_rows);

}  // namespace hdg
