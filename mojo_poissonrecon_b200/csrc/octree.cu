// Morton codes and the breadth-first flat octree on the device.
//
// Reference: src/capi.mojo:62-99 (codes), python/mojo_poissonrecon/core.py:86-127
// (per-level np.unique, breadth-first concatenation, parent/child links,
// point_leaf).  Here: leaf codes are radix-sorted once; because a level-l code
// is the leaf code shifted right by 3*(depth-l), the sorted leaf order is also
// sorted order at every level.  For sorted position i, L_i = the shallowest
// level at which its code differs from position i-1 (0 for i = 0, depth+1 for
// an identical leaf).  Position i starts a new level-l node iff L_i <= l, so a
// prefix count of (L_i <= l) numbers the level's nodes in ascending code
// order, exactly np.unique's order, and the level-(l-1) count at the same
// position is the parent.
//
// All levels at once: a tile of 1,024 positions counts its starts per level, one block
// per level scans the tiles, and the emission ranks a warp's positions by one ballot
// per level.  A node's first child starts at the same position, so child_start is a
// rank too, and the children end where the next node's begin: no atomics.  Bound by
// launches and latency (a million points at depth 10: flags, scan and emission level
// by level 250 us in 66 launches, now 40 in 4; the whole call 711 -> 256 us).
#include "radix_sort.cuh"

namespace pb {

// Per-level child index chain, capi.mojo:72-99 (integer conversion truncates
// toward zero, then clamps to [0, 2^level - 1]).
__device__ __forceinline__ int64_t level_cell(double v, int64_t scale) {
    int64_t i = (int64_t)(v * (double)scale);
    if (i < 0) i = 0;
    if (i >= scale) i = scale - 1;
    return i;
}

__global__ void octree_codes_kernel(const double* __restrict__ points, int64_t count, int depth,
                                    int64_t* __restrict__ codes) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    double x = points[3 * i], y = points[3 * i + 1], z = points[3 * i + 2];
    int64_t code = 0;
    int64_t* out = codes + i * (depth + 1);
    out[0] = 0;
    for (int d = 0; d < depth; ++d) {
        int64_t scale = (int64_t)1 << (d + 1);
        int64_t child = (level_cell(x, scale) & 1) | ((level_cell(y, scale) & 1) << 1) |
                        ((level_cell(z, scale) & 1) << 2);
        code = (code << 3) | child;
        out[d + 1] = code;
    }
}

// The low bits of v two places apart: bit k goes to bit 3 k.
__device__ __forceinline__ uint32_t spread(uint32_t v, uint32_t) {  // 10 bits
    v = (v | v << 16) & 0x030000ffu;
    v = (v | v << 8) & 0x0300f00fu;
    v = (v | v << 4) & 0x030c30c3u;
    return (v | v << 2) & 0x09249249u;
}
__device__ __forceinline__ uint64_t spread(uint64_t v, uint64_t) {  // 21 bits
    v = (v | v << 32) & 0x001f00000000ffffull;
    v = (v | v << 16) & 0x001f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    return (v | v << 2) & 0x1249249249249249ull;
}

// Leaf codes.  Scaling by a power of two is exact, so a level's cell is the deepest
// cell shifted right (and clamping commutes with the shift): one conversion per
// coordinate instead of one per level.  *outside (optional) counts points that are not
// finite or not in [0, 1]^3.
template <typename K>
__global__ void leaf_keys_kernel(const double* __restrict__ points, int64_t count, int depth, K* __restrict__ keys,
                                 uint32_t* __restrict__ vals, unsigned long long* __restrict__ outside) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool bad = false;
    if (i < count) {
        const double scale = (double)((int64_t)1 << depth), last = scale - 1.0;
        K code = 0;
#pragma unroll
        for (int axis = 0; axis < 3; ++axis) {
            const double v = points[3 * i + axis];
            bad |= !(v >= 0.0 && v <= 1.0);
            const uint32_t cell = (uint32_t)fmin(fmax(v * scale, 0.0), last);  // a NaN counts as 0, as level_cell's does
            code |= spread((K)cell, K()) << axis;
        }
        keys[i] = code;
        vals[i] = (uint32_t)i;
    }
    if (outside) {
        const int any = __syncthreads_count(bad);
        if (any && threadIdx.x == 0) atomicAdd(outside, (unsigned long long)any);
    }
}

constexpr int kLevels = 20;   // depth + 1 at most
constexpr int kTile = 1024;   // positions per block, one per thread
constexpr int kTileWarps = kTile / 32;

// L_i, and per level the tile's positions with L_i <= level: counts[level * tiles + tile].
template <typename K>
__global__ void __launch_bounds__(kTile) split_level_kernel(const K* __restrict__ keys, int64_t count, int depth,
                                                            uint8_t* __restrict__ split, uint32_t* __restrict__ counts,
                                                            uint32_t tiles) {
    __shared__ unsigned int hist[32];
    if (threadIdx.x < 32) hist[threadIdx.x] = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * kTile + threadIdx.x;
    int level = depth + 1;
    if (i < count) {
        if (i == 0) {
            level = 0;
        } else {
            const uint64_t diff = (uint64_t)(keys[i] ^ keys[i - 1]);
            if (diff) level = depth - (63 - __clzll((long long)diff)) / 3;
        }
        split[i] = (uint8_t)level;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, level);
    if (level <= depth && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&hist[level], (unsigned)__popc(peers));
    __syncthreads();
    if (threadIdx.x <= depth) {
        unsigned run = 0;
        for (int l = 0; l <= (int)threadIdx.x; ++l) run += hist[l];
        counts[(int64_t)threadIdx.x * tiles + blockIdx.x] = run;
    }
}

// One block per level: its nodes in earlier tiles, in place; level_counts[level].
__global__ void __launch_bounds__(kScanThreads) level_scan_kernel(uint32_t* __restrict__ counts, uint32_t tiles,
                                                                  int64_t* __restrict__ level_counts) {
    const uint32_t nodes = scan_row(counts + (int64_t)blockIdx.x * tiles, tiles);
    if (threadIdx.x == 0) level_counts[blockIdx.x] = (int64_t)nodes;
}

// First node of each level, and the total at [depth + 1].
__device__ __forceinline__ void level_offsets(const int64_t* __restrict__ level_counts, int depth, int64_t* offsets) {
    if (threadIdx.x == 0) {
        int64_t run = 0;
        for (int l = 0; l <= depth; ++l) {
            offsets[l] = run;
            run += level_counts[l];
        }
        offsets[depth + 1] = run;
    }
    __syncthreads();
}

// morton, parent and child_start of every node that a tile's positions start; point_leaf.
template <typename K>
__global__ void __launch_bounds__(kTile) emit_nodes_kernel(const K* __restrict__ keys, const uint32_t* __restrict__ perm,
                                                           const uint8_t* __restrict__ split, int64_t count, int depth,
                                                           const int64_t* __restrict__ level_counts,
                                                           const uint32_t* __restrict__ tile_starts, uint32_t tiles,
                                                           int64_t* __restrict__ morton, int64_t* __restrict__ parent,
                                                           int64_t* __restrict__ child_start,
                                                           int64_t* __restrict__ point_leaf) {
    __shared__ int64_t offsets[kLevels + 1];
    __shared__ uint32_t before[kLevels][kTileWarps];  // nodes of a level ahead of a warp's first position
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int64_t i = (int64_t)blockIdx.x * kTile + threadIdx.x;
    const int s = i < count ? split[i] : depth + 1;
    const int top = (int)__reduce_min_sync(0xffffffffu, (unsigned)s);  // the warp starts no node above this level
    if (lane < top && lane <= depth) before[lane][warp] = 0;
    for (int l = top; l <= depth; ++l) {
        const unsigned starts = __ballot_sync(0xffffffffu, s <= l);
        if (lane == 0) before[l][warp] = __popc(starts);
    }
    level_offsets(level_counts, depth, offsets);
    if (warp <= depth) {  // a warp per level: exclusive over the tile's warps
        const uint32_t v = before[warp][lane];
        uint32_t run = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t w = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += w;
        }
        before[warp][lane] = tile_starts[(int64_t)warp * tiles + blockIdx.x] + run - v;
    }
    __syncthreads();
    // the node of level l that position i starts or lies in; -1 before level 0
    auto node_at = [&](int l) -> int64_t {
        const unsigned starts = __ballot_sync(0xffffffffu, s <= l);
        return offsets[l] + before[l][warp] + __popc(starts & below) + (s <= l) - 1;
    };
    const K key = i < count ? keys[i] : K(0);
    int64_t up = top > 0 ? node_at(top - 1) : -1, node = top <= depth ? node_at(top) : -1;
    for (int l = top; l <= depth; ++l) {
        const int64_t down = l < depth ? node_at(l + 1) : -1;
        if (s <= l) {
            morton[node] = (int64_t)(key >> (3 * (depth - l)));
            parent[node] = up;
            child_start[node] = down;
        }
        up = node;
        node = down;
    }
    if (i < count) point_leaf[perm[i]] = up;
}

// node_depth, and child_count from where the next node's children start.
__global__ void __launch_bounds__(256) finish_nodes_kernel(const int64_t* __restrict__ level_counts, int depth,
                                                           const int64_t* __restrict__ child_start,
                                                           int64_t* __restrict__ node_depth,
                                                           int64_t* __restrict__ child_count) {
    __shared__ int64_t offsets[kLevels + 1];
    level_offsets(level_counts, depth, offsets);
    const int64_t leaves = offsets[depth], nodes = offsets[depth + 1];
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < nodes; i += (int64_t)gridDim.x * 256) {
        int level = depth;
        while (i < offsets[level]) --level;
        node_depth[i] = level;
        child_count[i] = i < leaves ? (i + 1 < leaves ? child_start[i + 1] : nodes) - child_start[i] : 0;
    }
}

// Codes of up to 10 levels fit 32 bits: half the sort's bytes.
static bool narrow_keys(int64_t depth) { return depth <= 10; }

struct OctreeWork {
    uint64_t *keys, *keys_alt;  // uint32_t where narrow
    uint32_t *vals, *vals_alt;
    uint8_t* split;
    uint32_t* counts;
    uint32_t tiles;
};

static OctreeWork octree_carve(Workspace& w, int64_t count) {
    OctreeWork o;
    o.keys = w.take<uint64_t>(count);
    o.keys_alt = w.take<uint64_t>(count);
    o.vals = w.take<uint32_t>(count);
    o.vals_alt = w.take<uint32_t>(count);
    o.split = w.take<uint8_t>(count);
    o.tiles = (uint32_t)((count + kTile - 1) / kTile);
    o.counts = w.take<uint32_t>((size_t)o.tiles * kLevels);
    return o;
}

static size_t octree_ws_bytes(int64_t count) {
    return measure([&](Workspace& w) {
        octree_carve(w, count);
        radix_carve<uint64_t>(w, count);
    });
}

static int check_octree_args(int64_t count, int64_t depth) {
    if (count < 1) return fail(PB_ERR_INVALID, "octree: point_count must be >= 1 (got %lld)", (long long)count);
    if (count > 0xFFFFFFFFll) return fail(PB_ERR_INVALID, "octree: point_count must be < 2^32");
    if (depth < 0 || depth > 19) return fail(PB_ERR_INVALID, "octree: depth must be between 0 and 19");
    return PB_OK;
}

}  // namespace pb

using namespace pb;

extern "C" int pb_octree_codes_f64(const double* points, int64_t point_count, int64_t depth, int64_t* codes,
                                   void* stream) {
    if (point_count < 0) return fail(PB_ERR_INVALID, "octree codes: negative point_count");
    if (depth < 0 || depth > 19) return fail(PB_ERR_INVALID, "octree codes: depth must be between 0 and 19");
    if (point_count == 0) return PB_OK;
    if (!points || !codes) return fail(PB_ERR_INVALID, "octree codes: null buffer");
    octree_codes_kernel<<<blocks_for(point_count, 256), 256, 0, (cudaStream_t)stream>>>(points, point_count,
                                                                                        (int)depth, codes);
    PB_CHECK_LAUNCH("octree_codes_kernel");
    return PB_OK;
}

extern "C" size_t pb_octree_workspace_size(int64_t point_count, int64_t depth) {
    (void)depth;
    return octree_ws_bytes(point_count < 1 ? 1 : point_count);
}

template <typename K>
static int octree_count(const double* points, int64_t count, int depth, int64_t* level_counts, int64_t* outside,
                        const OctreeWork& o, Workspace sort_ws, cudaStream_t s) {
    K *keys = (K*)o.keys, *keys_alt = (K*)o.keys_alt;
    if (outside) PB_CHECK_CUDA(cudaMemsetAsync(outside, 0, sizeof(int64_t), s), "octree outside");
    leaf_keys_kernel<K><<<blocks_for(count, 256), 256, 0, s>>>(points, count, depth, keys, o.vals,
                                                               (unsigned long long*)outside);
    PB_CHECK_LAUNCH("leaf_keys_kernel");
    bool in_alt = false;
    PB_TRY(radix_sort_pairs<K>(keys, o.vals, keys_alt, o.vals_alt, count, 3 * depth, &in_alt, sort_ws, s));
    split_level_kernel<K><<<o.tiles, kTile, 0, s>>>(in_alt ? keys_alt : keys, count, depth, o.split, o.counts, o.tiles);
    PB_CHECK_LAUNCH("split_level_kernel");
    level_scan_kernel<<<depth + 1, kScanThreads, 0, s>>>(o.counts, o.tiles, level_counts);
    PB_CHECK_LAUNCH("level_scan_kernel");
    return PB_OK;
}

// *outside (device, optional): points that are not finite or not in [0, 1]^3.
extern "C" int pb_octree_count_checked(const double* points, int64_t point_count, int64_t depth, int64_t* level_counts,
                                       int64_t* outside, void* workspace, size_t workspace_bytes, void* stream) {
    PB_TRY(check_octree_args(point_count, depth));
    if (!points || !level_counts) return fail(PB_ERR_INVALID, "octree count: null buffer");
    if (!workspace || workspace_bytes < octree_ws_bytes(point_count))
        return fail(PB_ERR_WORKSPACE, "octree count: workspace needs %zu bytes", octree_ws_bytes(point_count));
    Workspace w(workspace, workspace_bytes);
    const OctreeWork o = octree_carve(w, point_count);
    cudaStream_t s = (cudaStream_t)stream;
    return narrow_keys(depth)
               ? octree_count<uint32_t>(points, point_count, (int)depth, level_counts, outside, o, w, s)
               : octree_count<uint64_t>(points, point_count, (int)depth, level_counts, outside, o, w, s);
}

extern "C" int pb_octree_count(const double* points, int64_t point_count, int64_t depth, int64_t* level_counts,
                               void* workspace, size_t workspace_bytes, void* stream) {
    return pb_octree_count_checked(points, point_count, depth, level_counts, nullptr, workspace, workspace_bytes,
                                   stream);
}

extern "C" int pb_octree_emit(int64_t point_count, int64_t depth, const int64_t* level_counts, int64_t node_count,
                              int64_t* node_depth, int64_t* morton, int64_t* parent, int64_t* child_start,
                              int64_t* child_count, int64_t* point_leaf, void* workspace, size_t workspace_bytes,
                              void* stream) {
    PB_TRY(check_octree_args(point_count, depth));
    if (!level_counts || !node_depth || !morton || !parent || !child_start || !child_count || !point_leaf)
        return fail(PB_ERR_INVALID, "octree emit: null buffer");
    if (node_count < depth + 1) return fail(PB_ERR_INVALID, "octree emit: node_count too small");
    if (!workspace || workspace_bytes < octree_ws_bytes(point_count))
        return fail(PB_ERR_WORKSPACE, "octree emit: workspace needs %zu bytes", octree_ws_bytes(point_count));
    cudaStream_t s = (cudaStream_t)stream;
    Workspace w(workspace, workspace_bytes);
    const OctreeWork o = octree_carve(w, point_count);
    const int passes = (int)((3 * depth + 7) / 8);
    const bool in_alt = point_count > 1 && (passes & 1);
    const void* keys = in_alt ? o.keys_alt : o.keys;
    const uint32_t* perm = in_alt ? o.vals_alt : o.vals;
    if (narrow_keys(depth))
        emit_nodes_kernel<uint32_t><<<o.tiles, kTile, 0, s>>>((const uint32_t*)keys, perm, o.split, point_count,
                                                              (int)depth, level_counts, o.counts, o.tiles, morton,
                                                              parent, child_start, point_leaf);
    else
        emit_nodes_kernel<uint64_t><<<o.tiles, kTile, 0, s>>>((const uint64_t*)keys, perm, o.split, point_count,
                                                              (int)depth, level_counts, o.counts, o.tiles, morton,
                                                              parent, child_start, point_leaf);
    PB_CHECK_LAUNCH("emit_nodes_kernel");
    const int64_t blocks = (node_count + 255) / 256;
    finish_nodes_kernel<<<(unsigned)(blocks < 16 * kSMs ? blocks : 16 * kSMs), 256, 0, s>>>(
        level_counts, (int)depth, child_start, node_depth, child_count);
    PB_CHECK_LAUNCH("finish_nodes_kernel");
    return PB_OK;
}
