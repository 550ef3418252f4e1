// Occupancy words of a solve: where the screen, and the screen or the right-hand
// side, are not zero on the finest grid.
//
// Both are zero away from the samples (257^3, a million points: the screen at 2 % of
// the nodes), so the passes of the FP32-preconditioned solver read them only
// where they are not.  One bit covers 32 nodes of a row, and a word the 32 planes
// 32 c .. 32 c + 31 of those nodes, so that threads that march down z load one or
// two words for their whole march.  Two maps one after another in one buffer, word
// (c, y, x / 32) of each: where the screen is not zero, and where it or the
// right-hand side is not.
// A value with any bit set counts (a NaN, a negative zero), so skipping a read
// changes no bit of a result.
#pragma once

#include <stdint.h>

namespace pb {

struct Occupancy {
    int n;
    __host__ __device__ __forceinline__ int chunks() const { return (n + 31) >> 5; }
    __host__ __device__ __forceinline__ int tiles() const { return (n + 31) >> 5; }
    __host__ __device__ __forceinline__ int64_t chunk() const { return (int64_t)n * tiles(); }
    __host__ __device__ __forceinline__ int64_t map_words() const { return chunks() * chunk(); }
    __host__ __device__ __forceinline__ int64_t words() const { return 2 * map_words(); }
    // within a chunk
    __host__ __device__ __forceinline__ uint32_t at(int x, int y) const { return (uint32_t)y * tiles() + (x >> 5); }
};

__host__ __device__ __forceinline__ const uint32_t* screen_map(const void* occupancy) {
    return (const uint32_t*)occupancy;
}
__host__ __device__ __forceinline__ const uint32_t* either_map(const void* occupancy, int n) {
    return occupancy ? (const uint32_t*)occupancy + Occupancy{n}.map_words() : nullptr;
}

// The bits of planes z0 .. z0 + 31 at (x, y); all set without a map.
__device__ __forceinline__ uint32_t plane_bits(const uint32_t* __restrict__ map, int n, int x, int y, int z0) {
    if (!map) return 0xffffffffu;
    const Occupancy o{n};
    const uint32_t* word = map + (z0 >> 5) * o.chunk() + o.at(x, y);
    return __funnelshift_r(word[0], ((z0 >> 5) + 1) * 32 < n ? word[o.chunk()] : 0u, z0 & 31);
}

// Whether the five planes, rows and x around (x, y, z), all inside the grid, have none
// (false without a map; a whole word's 32 nodes count where x reaches one).
__device__ __forceinline__ bool five_cubed_empty(const uint32_t* __restrict__ map, int n, int x, int y, int z) {
    if (!map) return false;
    const Occupancy o{n};
    const int z0 = z - 2, shift = z0 & 31;
    const uint32_t low = 0x1fu << shift, high = shift > 27 ? 0x1fu >> (32 - shift) : 0u;
    const bool two = (x - 2) >> 5 != (x + 2) >> 5;
    const uint32_t* word = map + (z0 >> 5) * o.chunk() + o.at(x - 2, y - 2);
    uint32_t any = 0;
#pragma unroll
    for (int row = 0; row < 5; ++row, word += o.tiles()) {
        any |= word[0] & low;
        if (two) any |= word[1] & low;
        if (high) {
            any |= word[o.chunk()] & high;
            if (two) any |= word[o.chunk() + 1] & high;
        }
    }
    return any == 0;
}

}  // namespace pb
