// The determinant table: open addressing over (alpha group, beta string), one-word strings.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace risq {

// Hash of (alpha group, beta string) (splitmix64 finaliser).
__device__ __forceinline__ uint64_t det_hash(uint32_t g, uint64_t beta) {
    uint64_t h = beta * 0x9E3779B97F4A7C15ull ^ ((uint64_t)(g + 1) * 0xC2B2AE3D27D4EB4Full);
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 29;
    return h;
}

// 2^bits slots {beta low, beta high, alpha group, internal index}, index -1 = empty.
struct DetTable {
    const int4* slots;
    int bits;
    // internal index of the determinant (alpha group g, beta string beta), or -1
    __device__ __forceinline__ int find(int g, uint64_t beta) const {
        const uint32_t mask = (1u << bits) - 1u;
        uint32_t slot = (uint32_t)(det_hash((uint32_t)g, beta) >> (64 - bits));
        const int lo = (int)(uint32_t)beta, hi = (int)(uint32_t)(beta >> 32);
        for (uint32_t t = 0; t <= mask; t++) {
            const int4 e = __ldg(slots + slot);
            if (e.w < 0) return -1;
            if (e.x == lo && e.y == hi && e.z == g) return e.w;
            slot = (slot + 1) & mask;
        }
        return -1;
    }
};

}  // namespace risq
