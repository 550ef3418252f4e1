// Stable LSD radix sort of (key, uint32 value) pairs, 8-bit digits.
//
// Per digit pass: (1) per-tile digit histograms, (2) one block per digit scans its
// tiles' counts and totals them, (3) each tile adds the digits' own starts (a scan of
// the 256 totals, made again by every block), ranks its items stably — warps take 32
// consecutive items per round and rank equal digits with __match_any_sync —
// stages them in shared memory in digit order and writes them out in runs.
// Three launches a pass; the device-wide scan of all (digit, tile) counts that step 2
// replaces took three by itself (a million keys: 12 us a pass, now 3).
#pragma once

#include "scan.cuh"

namespace pb {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Items per lane, ROUNDS: a tile holds 256 * ROUNDS consecutive items, each warp 32 * ROUNDS of
// them.  A tile's rounds run one after another, so small sorts take 4 (20,000 items:
// 4.3 us a scatter instead of 5.9, 2.9 us a histogram instead of 3.8); beyond 2^20 items
// both fill the GPU, and 8 halve the counts.  Octree count at depth 10 (four passes of
// 32-bit keys), us with 4 / 8 rounds: 100,000 points 75 / 91, 2^18 82 / 92, 2^19 105 /
// 103, 2^20 130 / 130, 1.5 million 167 / 142, 2^22 344 / 311, 2^24 1,168 / 1,002; with
// 64-bit keys (depth 19) 131 / 163, 147 / 164, 186 / 183, 249 / 245, 311 / 281, 661 / 580.
inline int sort_rounds(int64_t count) { return count <= (1 << 20) ? 4 : 8; }
inline int64_t sort_tiles(int64_t count) {
    const int64_t tile = (int64_t)kSortThreads * sort_rounds(count);
    return (count + tile - 1) / tile;
}
constexpr unsigned kNoDigit = 256u;

template <typename K, int ROUNDS>
__global__ void __launch_bounds__(kSortThreads) radix_histogram(const K* __restrict__ keys, int64_t count,
                                                                int shift, uint32_t* __restrict__ counts,
                                                                uint32_t tiles) {
    constexpr int kItems = kSortThreads * ROUNDS;
    __shared__ uint32_t hist[256];
    hist[threadIdx.x] = 0;
    __syncthreads();
    int64_t base = (int64_t)blockIdx.x * kItems;
    for (int k = threadIdx.x; k < kItems; k += kSortThreads) {
        int64_t i = base + k;
        if (i < count) atomicAdd(&hist[(unsigned)(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    counts[(int64_t)threadIdx.x * tiles + blockIdx.x] = hist[threadIdx.x];
}

// counts[digit * tiles + tile] -> the digit's items in earlier tiles; totals[digit].
static __global__ void __launch_bounds__(kScanThreads) radix_scan_digits(uint32_t* __restrict__ counts, uint32_t tiles,
                                                                        uint32_t* __restrict__ totals) {
    const uint32_t before = scan_row(counts + (int64_t)blockIdx.x * tiles, tiles);
    if (threadIdx.x == 0) totals[blockIdx.x] = before;
}

template <typename K, int ROUNDS>
__global__ void __launch_bounds__(kSortThreads) radix_scatter(const K* __restrict__ keys_in,
                                                              const uint32_t* __restrict__ vals_in,
                                                              K* __restrict__ keys_out,
                                                              uint32_t* __restrict__ vals_out, int64_t count,
                                                              int shift, const uint32_t* __restrict__ offsets,
                                                              const uint32_t* __restrict__ totals, uint32_t tiles) {
    constexpr int kItems = kSortThreads * ROUNDS;
    __shared__ uint32_t warp_hist[kSortWarps][256];
    __shared__ uint32_t digit_start[256], digit_out[256];
    __shared__ uint32_t warp_sums[32];
    __shared__ K s_keys[kItems];
    __shared__ uint32_t s_vals[kItems];

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kSortWarps * 256; k += kSortThreads) (&warp_hist[0][0])[k] = 0;
    __syncthreads();

    const int64_t tile_base = (int64_t)blockIdx.x * kItems;
    const int64_t warp_base = tile_base + (int64_t)warp * (32 * ROUNDS);
    const unsigned lt_mask = (1u << lane) - 1u;
    K key[ROUNDS];
    uint32_t val[ROUNDS];
    uint32_t rank[ROUNDS];
    unsigned dig[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        int64_t i = warp_base + r * 32 + lane;
        bool valid = i < count;
        key[r] = valid ? keys_in[i] : K(0);
        val[r] = valid ? vals_in[i] : 0u;
        unsigned d = valid ? ((unsigned)(key[r] >> shift) & 255u) : kNoDigit;
        dig[r] = d;
        unsigned peers = __match_any_sync(0xffffffffu, d);
        int leader = __ffs(peers) - 1;
        uint32_t before = 0;
        if (lane == leader && d != kNoDigit) {
            before = warp_hist[warp][d];
            warp_hist[warp][d] = before + __popc(peers);
        }
        before = __shfl_sync(0xffffffffu, before, leader);
        rank[r] = before + __popc(peers & lt_mask);
        __syncwarp();
    }
    __syncthreads();
    // Per digit: exclusive offsets of the warps, then the tile's digit totals.
    uint32_t digit_total = 0;
    {
        const unsigned d = threadIdx.x;  // kSortThreads == 256 digits
        uint32_t run = 0;
#pragma unroll
        for (int w = 0; w < kSortWarps; ++w) {
            uint32_t t = warp_hist[w][d];
            warp_hist[w][d] = run;
            run += t;
        }
        digit_total = run;
    }
    uint32_t all, tile_total;
    // where the digit's items of this tile go, less their first place within the tile
    digit_out[threadIdx.x] = block_exclusive_scan<uint32_t>(totals[threadIdx.x], warp_sums, all) +
                             offsets[(int64_t)threadIdx.x * tiles + blockIdx.x];
    uint32_t start = block_exclusive_scan<uint32_t>(digit_total, warp_sums, tile_total);
    digit_start[threadIdx.x] = start;
    digit_out[threadIdx.x] -= start;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; ++r) {
        if (dig[r] == kNoDigit) continue;
        uint32_t pos = digit_start[dig[r]] + warp_hist[warp][dig[r]] + rank[r];
        s_keys[pos] = key[r];
        s_vals[pos] = val[r];
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < tile_total; j += kSortThreads) {
        K k = s_keys[j];
        unsigned d = (unsigned)(k >> shift) & 255u;
        const uint32_t out = digit_out[d] + j;  // below count <= 2^32 - 1
        keys_out[out] = k;
        vals_out[out] = s_vals[j];
    }
}

template <typename K>
void radix_carve(Workspace& ws, int64_t count) {
    const int64_t tiles = sort_tiles(count);
    ws.take<uint32_t>(tiles * 256);
    ws.take<uint32_t>(256);
}

// Sorts (keys, vals) by bits [0, bits) of the key, stably.  Ping-pongs between
// the primary and alternate buffers; *result_in_alt says where the result is.
template <typename K>
int radix_sort_pairs(K* keys, uint32_t* vals, K* keys_alt, uint32_t* vals_alt, int64_t count, int bits,
                     bool* result_in_alt, Workspace& ws, cudaStream_t s) {
    *result_in_alt = false;
    if (count <= 1 || bits <= 0) return PB_OK;
    if (count > (int64_t)0xFFFFFFFFll) return fail(PB_ERR_INVALID, "radix sort: too many items");
    const int64_t tiles = sort_tiles(count);
    uint32_t* counts = ws.take<uint32_t>(tiles * 256);
    uint32_t* totals = ws.take<uint32_t>(256);
    if (!ws.fits()) return fail(PB_ERR_WORKSPACE, "radix sort workspace too small");
    K* src_k = keys;
    uint32_t* src_v = vals;
    K* dst_k = keys_alt;
    uint32_t* dst_v = vals_alt;
    for (int shift = 0; shift < bits; shift += 8) {
        auto histogram = sort_rounds(count) == 4 ? radix_histogram<K, 4> : radix_histogram<K, 8>;
        auto scatter = sort_rounds(count) == 4 ? radix_scatter<K, 4> : radix_scatter<K, 8>;
        histogram<<<(unsigned)tiles, kSortThreads, 0, s>>>(src_k, count, shift, counts, (uint32_t)tiles);
        PB_CHECK_LAUNCH("radix_histogram");
        radix_scan_digits<<<256, kScanThreads, 0, s>>>(counts, (uint32_t)tiles, totals);
        PB_CHECK_LAUNCH("radix_scan_digits");
        scatter<<<(unsigned)tiles, kSortThreads, 0, s>>>(src_k, src_v, dst_k, dst_v, count, shift, counts, totals,
                                                         (uint32_t)tiles);
        PB_CHECK_LAUNCH("radix_scatter");
        K* tk = src_k; src_k = dst_k; dst_k = tk;
        uint32_t* tv = src_v; src_v = dst_v; dst_v = tv;
        *result_in_alt = !*result_in_alt;
    }
    return PB_OK;
}

}  // namespace pb
