// packed16.cuh -- two 16-bit values in one register: packing and byte permutes.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gba {

__device__ __forceinline__ uint32_t pack2(int lo, int hi)
{
    return (uint32_t(lo) & 0xffffu) | (uint32_t(hi) << 16);
}
__device__ __forceinline__ int lo16(uint32_t x) { return int(int16_t(x & 0xffffu)); }
__device__ __forceinline__ int hi16(uint32_t x) { return int(int16_t(x >> 16)); }

__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel)
{
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// Selector half for a row code v (3 bits): byte nibble v, then 8|v (sign replicate).
__device__ __forceinline__ uint32_t vsel_of(uint32_t byte)
{
    const uint32_t a = byte & 7u, b = (byte >> 4) & 7u;
    return a | ((a | 8u) << 4) | (b << 8) | ((b | 8u) << 12);
}

}  // namespace gba
