// Two-pass trilinear splat, bit-identical to the serial reference.
//
// Reference: src/capi.mojo:104-224.  The reference adds each sample's eight
// corner weights into the grids in point order; floating-point addition is not
// associative, so atomics would change the last bits.  Here a stable radix sort
// groups the points by cell, keeping point order inside each cell.  A grid node
// is touched by the points of the (at most) eight cells around it, eight lists
// sorted by point: one thread per touched node merges them, which visits the
// node's contributions in point order and adds them from the node's current
// value: the same additions, in the same order, as the reference.  The merge
// leaves the node's contributions (sorted place of the point, corner) as a list,
// which pass 2 (both passes address the same eight nodes per sample) and the
// attribute sums then only walk.  Where points crowd, a node's long list is put in
// order and summed by many threads (below: long lists).
//
// Against one record per (point, corner) sorted by node and five dense grids
// (B200, 1M noisy points at depth 8): the sort handles 1M keys instead of 8M (370 ->
// 85 us), no record is written, gathered or compacted, and with the vector field at
// the touched nodes only, points to density, screen and rhs take 620 us instead of 1,420.
//
// Compiled with -fmad=false: every product and sum rounds as written.
#include <algorithm>

#include "radix_sort.cuh"

namespace pb {

__device__ __forceinline__ double norm3(double x, double y, double z) {  // capi.mojo:51-59
    double scale = fmax(fabs(x), fmax(fabs(y), fabs(z)));
    if (scale == 0.0) return 0.0;
    double sx = x / scale, sy = y / scale, sz = z / scale;
    return scale * sqrt(sx * sx + sy * sy + sz * sz);
}

__device__ __forceinline__ double clamp01(double v) {  // min(max(v, 0), 1)
    double m = v > 0.0 ? v : 0.0;
    return m < 1.0 ? m : 1.0;
}

// Pass-1 base cell and fractions (capi.mojo:139-162).
__device__ __forceinline__ void pass1_cell(double p, int64_t res, int64_t& i, double& f) {
    double g = p * (double)res;
    i = (int64_t)g;
    if (i < 0) i = 0;
    if (i >= res) {
        i = res - 1;
        g = (double)res;
    }
    f = g - (double)i;
}

// Pass-2 / iso-value base cell and fractions (capi.mojo:187-195, :771-779).
__device__ __forceinline__ void pass2_cell(double p, int64_t res, int64_t& i, double& f) {
    double g = p * (double)res;
    int64_t t = (int64_t)g;
    i = t < 0 ? 0 : (t > res - 1 ? res - 1 : t);
    f = clamp01(g - (double)i);
}

// A sorted point: its fractions in its cell and its sample weight (0: rejected, capi.mojo:132-133);
// its unit normal and, for pass 2, its density factor.
struct alignas(32) Frac {
    double x, y, z, weight;
};
struct alignas(32) Unit {
    double x, y, z, factor;
};

// One 32-byte load each: the lists visit points out of order, and four 8-byte loads of a warp would
// look up four times as many sectors (L1 lookups bound the walks: pass 2 over 8M contributions 199 -> 125 us).
template <typename T>
__device__ __forceinline__ T load32(const T* p) {
    static_assert(sizeof(T) == 32, "one 256-bit load");
    T v;
    asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
        : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(reinterpret_cast<double*>(&v)[3])
        : "l"(p));
    return v;
}

// Trilinear weight of corner c times the sample weight (capi.mojo:163-170).
__device__ __forceinline__ double corner_weight(double fx, double fy, double fz, double weight, int c) {
    const double wz = (c & 4) ? fz : 1.0 - fz;
    const double wy = (c & 2) ? fy : 1.0 - fy;
    const double wx = (c & 1) ? fx : 1.0 - fx;
    return wx * wy * wz * weight;
}

// Cell of every point (rejected ones in the last, where their zero weight adds nothing) and the
// accepted samples' number.
__global__ void __launch_bounds__(256) cell_keys_kernel(const double* __restrict__ points,
                                                        const double* __restrict__ normals, int64_t count, int64_t n,
                                                        uint32_t* __restrict__ keys, uint32_t* __restrict__ vals,
                                                        unsigned long long* __restrict__ accepted) {
    __shared__ unsigned int block_accepted;
    if (threadIdx.x == 0) block_accepted = 0;
    __syncthreads();
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool valid = false;
    if (p < count) {
        const int64_t c = n - 1;
        valid = !(norm3(normals[3 * p], normals[3 * p + 1], normals[3 * p + 2]) <= 0.0);  // capi.mojo:132-133
        int64_t ix = c - 1, iy = c - 1, iz = c - 1;
        double f;
        if (valid) {
            pass1_cell(points[3 * p], c, ix, f);
            pass1_cell(points[3 * p + 1], c, iy, f);
            pass1_cell(points[3 * p + 2], c, iz, f);
        }
        keys[p] = (uint32_t)((iz * c + iy) * c + ix);
        vals[p] = (uint32_t)p;
    }
    const unsigned ballot = __ballot_sync(0xffffffffu, valid);
    if ((threadIdx.x & 31) == 0 && ballot) atomicAdd(&block_accepted, __popc(ballot));
    __syncthreads();
    if (threadIdx.x == 0 && block_accepted) atomicAdd(accepted, (unsigned long long)block_accepted);
}

// Points in sorted order, and the flag of each cell's first.
__global__ void __launch_bounds__(256) gather_points_kernel(const double* __restrict__ points,
                                                            const double* __restrict__ normals, int64_t count,
                                                            int64_t n, int confidence,
                                                            const uint32_t* __restrict__ keys,
                                                            const uint32_t* __restrict__ vals,
                                                            Frac* __restrict__ frac, Unit* __restrict__ unit,
                                                            uint32_t* __restrict__ flag) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= count) return;
    flag[j] = j == 0 || keys[j - 1] != keys[j];
    const int64_t p = vals[j], c = n - 1;
    const double nx = normals[3 * p], ny = normals[3 * p + 1], nz = normals[3 * p + 2];
    const double length = norm3(nx, ny, nz);
    Frac f = {0.0, 0.0, 0.0, 0.0};
    Unit u = {0.0, 0.0, 0.0, 1.0};
    if (!(length <= 0.0)) {
        int64_t i;
        pass1_cell(points[3 * p], c, i, f.x);
        pass1_cell(points[3 * p + 1], c, i, f.y);
        pass1_cell(points[3 * p + 2], c, i, f.z);
        f.weight = confidence ? length : 1.0;
        u.x = nx / length;
        u.y = ny / length;
        u.z = nz / length;
    }
    frac[j] = f;
    if (unit) unit[j] = u;
}

// heads[r] = first sorted point of occupied cell r (heads[cells] = count); table[cell] = r + 1.
__global__ void __launch_bounds__(256) cell_table_kernel(const uint32_t* __restrict__ keys,
                                                         const uint32_t* __restrict__ rank, int64_t count,
                                                         const uint32_t* __restrict__ cells,
                                                         uint32_t* __restrict__ heads, uint32_t* __restrict__ table) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= count) return;
    if (j == 0 || keys[j - 1] != keys[j]) {
        heads[rank[j]] = (uint32_t)j;
        table[keys[j]] = rank[j] + 1;
    }
    if (j == 0) heads[*cells] = (uint32_t)count;
}

struct Cells {  // the occupied cells
    uint32_t n, c;
    FastDiv by_c, by_n;
    const uint32_t *table, *heads;
    // The occupied cell at (x, y, z) + 1, 0 where there is none (or no such cell).
    __device__ __forceinline__ uint32_t at(uint32_t x, uint32_t y, uint32_t z) const {
        return x < c && y < c && z < c ? table[(z * c + y) * c + x] : 0u;
    }
};

// Touched nodes: (occupied cell, corner) pairs whose cell is the first occupied one around the
// node.  A node's slot in the list and its place among the contributions come from counters, warp
// by warp: their order changes from run to run, the contents of a slot do not.  A thread takes a
// cell with its 27 neighbours (their lookups serve all eight corners, and consecutive cells of a
// row share sectors): bound by L1 lookups, 1M points at 257^3 71 us with a thread per corner, now 18.
struct Nodes {
    uint32_t *node, *base, *length;
    uint32_t* slot_of;  // dense node -> slot + 1 (may be null)
    uint32_t* counters;  // slots, contributions, units, long lists
    uint2* units;        // (slot, part) of the long lists, kUnit contributions each
    uint32_t* longs;     // slots of the long lists
    uint32_t long_over;  // a list is long beyond this many contributions (long_over_of)
};
constexpr uint32_t kUnit = 256;

// Where a list counts as long.  One thread per list waits for its loads, which only many
// lists side by side hide, and the larger the grid the more nodes a surface touches; a
// block per list costs a few microseconds however short the list.  Splat and assembly,
// us, with the line at 64 / 128 / 512: 100,000 points at 33^3 211 / 273 / 363; 200,000 at
// 65^3 329 / 279 / 277, a million 860 / 881 / 1,056; a million at 129^3 1,048 / 887 / 567,
// two million 1,788 / 1,744 / 1,021; at 257^3 four million 4,116 / 3,268 / 1,708.
constexpr uint32_t kLongOver = 64;  // the least of them
static uint32_t long_over_of(int64_t n) { return n <= 33 ? kLongOver : n <= 65 ? 128 : 512; }

__global__ void __launch_bounds__(128) touched_nodes_kernel(Cells g, const uint32_t* __restrict__ keys,
                                                            const uint32_t* __restrict__ cells, Nodes out) {
    const uint32_t total = *cells, stride = gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t - lane < total; t += stride) {
        uint32_t node = 0, points[27], owned = 0, sum = 0;  // points of the cells around; owned corners
        if (t < total) {
            const uint32_t cell = keys[g.heads[t]];
            const uint32_t row = g.by_c.div(cell), z = g.by_c.div(row), y = row - z * g.c, x = cell - row * g.c;
            node = (z * g.n + y) * g.n + x;
#pragma unroll
            for (int k = 0; k < 27; ++k) points[k] = g.at(x + (k % 3 - 1), y + (k / 3 % 3 - 1), z + (k / 9 - 1));
#pragma unroll
            for (int k = 0; k < 27; ++k)
                if (points[k]) points[k] = g.heads[points[k]] - g.heads[points[k] - 1];
#pragma unroll
            for (int corner = 0; corner < 8; ++corner) {
                // the cells around the corner's node, whose corner k it is; they ascend as k descends, and the
                // node is the cell's own if none occupied comes before it
                uint32_t length = 0, before = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const uint32_t v = points[((corner & 1) - (k & 1) + 1) + 3 * (((corner >> 1) & 1) - ((k >> 1) & 1) + 1) +
                                              9 * ((corner >> 2) - (k >> 2) + 1)];
                    length += v;
                    if (k > corner) before |= v;
                }
                if (before == 0) {
                    owned |= 1u << corner;
                    sum += length;
                }
            }
        }
        const uint32_t nodes = __popc(owned);
        uint32_t slots = nodes, contributions = sum;  // inclusive over the warp
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, slots, o), b = __shfl_up_sync(0xffffffffu, contributions, o);
            if (lane >= o) {
                slots += a;
                contributions += b;
            }
        }
        uint32_t slot0 = 0, base0 = 0;
        if (lane == 31 && slots) {
            slot0 = atomicAdd(out.counters, slots);
            base0 = atomicAdd(out.counters + 1, contributions);
        }
        uint32_t slot = __shfl_sync(0xffffffffu, slot0, 31) + slots - nodes;
        uint32_t base = __shfl_sync(0xffffffffu, base0, 31) + contributions - sum;
        if (owned)
#pragma unroll
            for (int corner = 0; corner < 8; ++corner)
                if (owned >> corner & 1u) {
                    uint32_t length = 0;
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        length += points[((corner & 1) - (k & 1) + 1) + 3 * (((corner >> 1) & 1) - ((k >> 1) & 1) + 1) +
                                         9 * ((corner >> 2) - (k >> 2) + 1)];
                    const uint32_t at = node + (corner & 1) + ((corner >> 1) & 1) * g.n + (corner >> 2) * g.n * g.n;
                    out.node[slot] = at;
                    out.base[slot] = base;
                    out.length[slot] = length;
                    if (out.slot_of) out.slot_of[at] = slot + 1;
                    if (length > out.long_over) {
                        out.longs[atomicAdd(out.counters + 3, 1u)] = slot;
                        const uint32_t parts = (length + kUnit - 1) / kUnit, first = atomicAdd(out.counters + 2, parts);
                        for (uint32_t part = 0; part < parts; ++part) out.units[first + part] = make_uint2(slot, part);
                    }
                    ++slot;
                    base += length;
                }
    }
}

constexpr uint32_t kPlaceBits = 29, kNone = 0xFFFFFFFFu;

// ---- long lists -------------------------------------------------------------------
// One thread's walk waits for its loads at every contribution, which many short lists
// hide and a long one does not (a million points at depth 3: lists of 30,000).  A long
// list is put in order by ranks: a contribution's place is the number of points before
// it in each of the eight sorted lists, all searched at once, a thread per contribution.
// Its sums keep the reference's order, one addition after another, but only the
// additions wait for each other: seven warps of a block read the contributions and form
// their values in shared memory a tile ahead of the threads that add them.
// Splat and assembly of a million points, one thread per list -> this: at depth 2 338 ->
// 4.1 ms, 3 82 -> 1.4, 4 18.3 -> 0.95, 5 4.5 -> 0.85; half of them in a thousandth of
// the surface, at depth 6, 468 -> 6.4.  What is left is the chain of additions of the
// longest list.

// Part unit.y of the list of slot unit.x.
__device__ __forceinline__ void rank_unit(const Cells& g, const Nodes& nodes, const uint32_t* __restrict__ order,
                                          uint32_t* __restrict__ list, uint2 unit) {
    const uint32_t node = nodes.node[unit.x], row = g.by_n.div(node), z = g.by_n.div(row), x = node - row * g.n,
                   y = row - z * g.n;
    uint32_t start[8], size[8], most = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const uint32_t r = g.at(x - (k & 1), y - ((k >> 1) & 1), z - (k >> 2));
        start[k] = r ? g.heads[r - 1] : 0u;
        size[k] = r ? g.heads[r] - start[k] : 0u;
        most = max(most, size[k]);
    }
    uint32_t left = unit.y * kUnit + threadIdx.x, place = kNone, corner = 0;  // of the lists one after another
#pragma unroll
    for (int k = 0; k < 8; ++k)
        if (place == kNone) {
            if (left < size[k]) {
                place = start[k] + left;
                corner = k;
            } else {
                left -= size[k];
            }
        }
    if (place == kNone) return;  // past the last list
    const uint32_t point = order[place];
    uint32_t before[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (uint32_t step = 0x80000000u >> __clz(most); step; step >>= 1)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t at = before[k] + step;
            if (at <= size[k] && order[start[k] + at - 1] < point) before[k] = at;
        }
    uint32_t rank = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) rank += before[k];
    list[nodes.base[unit.x] + rank] = place | corner << kPlaceBits;
}

constexpr int kAhead = 224;  // contributions of a tile: one per thread of the seven reading warps

// acc + the list's values of chain threadIdx.x, in order, in the first CHAINS threads (of 256);
// values(contribution, v): its value in each chain.
template <int CHAINS, typename Values>
__device__ __forceinline__ double add_in_order(const uint32_t* __restrict__ in, uint32_t length, double acc,
                                               Values&& values) {
    __shared__ double tiles[2][CHAINS][kAhead];
    const int reader = (int)threadIdx.x - 32;
    const uint32_t count = (length + kAhead - 1) / kAhead;
    for (uint32_t t = 0; t <= count; ++t) {  // tile t is read while tile t - 1 is added
        if (reader >= 0) {
            const uint32_t i = t * kAhead + reader;
            if (i < length) {
                double v[CHAINS];
                values(in[i], v);
#pragma unroll
                for (int c = 0; c < CHAINS; ++c) tiles[t & 1][c][reader] = v[c];
            }
        } else if (t > 0 && threadIdx.x < CHAINS) {
            const double* v = tiles[(t - 1) & 1][threadIdx.x];
            const uint32_t n = min((uint32_t)kAhead, length - (t - 1) * kAhead);
#pragma unroll 16
            for (uint32_t j = 0; j < n; ++j) acc += v[j];
        }
        __syncthreads();
    }
    return acc;
}

// Pass 1 (capi.mojo:171-172) of the long lists.
__global__ void __launch_bounds__(256) long_sums_kernel(Nodes nodes, const uint32_t* __restrict__ list,
                                                        const Frac* __restrict__ frac, double* __restrict__ density,
                                                        double* __restrict__ screen) {
    const uint32_t count = nodes.counters[3];
    for (uint32_t i = blockIdx.x; i < count; i += gridDim.x) {
        const uint32_t slot = nodes.longs[i];
        double* grid = threadIdx.x == 0 ? density : screen;
        const uint32_t node = nodes.node[slot];
        const double acc = add_in_order<2>(list + nodes.base[slot], nodes.length[slot],
                                           threadIdx.x < 2 ? grid[node] : 0.0, [&](uint32_t item, double (&v)[2]) {
                                               const Frac f = load32(frac + (item & ((1u << kPlaceBits) - 1u)));
                                               v[1] = corner_weight(f.x, f.y, f.z, f.weight, (int)(item >> kPlaceBits));
                                               v[0] = 2.0 * v[1];
                                           });
        if (threadIdx.x < 2) grid[node] = acc;
    }
}

// Merges each node's lists into its contributions, (sorted point | corner << 29) in point order,
// and, SUMS, adds pass 1 (capi.mojo:171-172): density += 2w, screen += w.  Cursors, current and next
// point of all eight lists stay in registers; the next point is read an addition ahead.  The last
// unit_blocks blocks rank the long lists: behind the others, they delay nothing where there are none
// (50,000 points at depth 6 173 -> 162 us; 159 without them).
template <bool SUMS>
__global__ void __launch_bounds__(256) merge_kernel(Cells g, Nodes nodes, const uint32_t* __restrict__ order,
                                                    const Frac* __restrict__ frac, uint32_t* __restrict__ list,
                                                    double* __restrict__ density, double* __restrict__ screen,
                                                    uint32_t unit_blocks) {
    const uint32_t merge_blocks = gridDim.x - unit_blocks;
    if (blockIdx.x >= merge_blocks) {
        const uint32_t units = nodes.counters[2];
        for (uint32_t u = blockIdx.x - merge_blocks; u < units; u += unit_blocks)
            rank_unit(g, nodes, order, list, nodes.units[u]);
        return;
    }
    const uint32_t count = nodes.counters[0], stride = merge_blocks * blockDim.x;
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < count; slot += stride) {
        const uint32_t length = nodes.length[slot];
        if (length > nodes.long_over) continue;
        const uint32_t node = nodes.node[slot], row = g.by_n.div(node), z = g.by_n.div(row), x = node - row * g.n,
                       y = row - z * g.n;
        uint32_t* __restrict__ out = list + nodes.base[slot];
        uint32_t cur[8], end[8], point[8], next[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t r = g.at(x - (k & 1), y - ((k >> 1) & 1), z - (k >> 2));
            cur[k] = r ? g.heads[r - 1] : 0u;
            end[k] = r ? g.heads[r] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            point[k] = cur[k] < end[k] ? order[cur[k]] : kNone;
            next[k] = cur[k] + 1 < end[k] ? order[cur[k] + 1] : kNone;
        }
        double d = 0.0, s = 0.0;
        if (SUMS) {
            d = density[node];
            s = screen[node];
        }
        for (uint32_t t = 0; t < length; ++t) {
            uint32_t least = point[0];
#pragma unroll
            for (int k = 1; k < 8; ++k) least = min(least, point[k]);
            uint32_t place = 0, corner = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
                if (point[k] == least) {
                    place = cur[k]++;
                    corner = k;
                    point[k] = next[k];
                    next[k] = cur[k] + 1 < end[k] ? order[cur[k] + 1] : kNone;
                }
            out[t] = place | corner << kPlaceBits;
            if (SUMS) {
                const Frac f = load32(frac + place);
                const double w = corner_weight(f.x, f.y, f.z, f.weight, (int)corner);
                d += 2.0 * w;
                s += w;
            }
        }
        if (SUMS) {
            density[node] = d;
            screen[node] = s;
        }
    }
}

// Pass 2, per sample (capi.mojo:176-209): the density factor from the pass-1 grid.
__global__ void __launch_bounds__(256) density_factor_kernel(int64_t count, int64_t n, const uint32_t* __restrict__ keys,
                                                             const Frac* __restrict__ frac, double samples_per_node,
                                                             const double* __restrict__ density,
                                                             Unit* __restrict__ unit) {
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= count) return;
    const uint32_t c = (uint32_t)(n - 1), cell = keys[j], row = cell / c, cz = row / c;
    const int64_t node = grid_index(cell - row * c, row - cz * c, cz, n);
    const Frac f = frac[j];
    const double fx = clamp01(f.x), fy = clamp01(f.y), fz = clamp01(f.z);
    double local = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double wz = (k & 4) ? fz : 1.0 - fz;
        const double wy = (k & 2) ? fy : 1.0 - fy;
        const double wx = (k & 1) ? fx : 1.0 - fx;
        local += density[node + ((k >> 2) * n + ((k >> 1) & 1)) * n + (k & 1)] * wx * wy * wz;
    }
    const double q = local / samples_per_node;
    unit[j].factor = 1.0 > q ? 1.0 : q;
}

// Pass 2 (capi.mojo:221-223): V -= n_hat * (w * res / factor), per node in point order, into dense
// grids or, COMPACT, into v[slot]; and the density divided by samples_per_node (core.py:255; COMPACT:
// only the touched nodes, 0 / samples_per_node being 0 elsewhere).  The last long_blocks blocks take the
// long lists.
template <bool COMPACT>
__global__ void __launch_bounds__(256) vector_kernel(Nodes nodes, const uint32_t* __restrict__ list,
                                                     const Frac* __restrict__ frac, const Unit* __restrict__ unit,
                                                     double res, double* __restrict__ vx, double* __restrict__ vy,
                                                     double* __restrict__ vz, double* __restrict__ density,
                                                     double samples_per_node, uint32_t long_blocks) {
    auto values = [&](uint32_t item, double (&v)[3]) {  // what a contribution takes from V
        const uint32_t place = item & ((1u << kPlaceBits) - 1u);
        const Frac f = load32(frac + place);
        const Unit u = load32(unit + place);
        const double w = corner_weight(clamp01(f.x), clamp01(f.y), clamp01(f.z), f.weight, (int)(item >> kPlaceBits));
        const double vw = w * res / u.factor;
        v[0] = u.x * vw;
        v[1] = u.y * vw;
        v[2] = u.z * vw;
    };
    const uint32_t walk_blocks = gridDim.x - long_blocks;
    if (blockIdx.x >= walk_blocks) {
        const uint32_t longs = nodes.counters[3];
        for (uint32_t i = blockIdx.x - walk_blocks; i < longs; i += long_blocks) {
            const uint32_t slot = nodes.longs[i], node = nodes.node[slot], at = COMPACT ? slot : node;
            double* grid = threadIdx.x == 0 ? vx : threadIdx.x == 1 ? vy : vz;
            const double acc = add_in_order<3>(list + nodes.base[slot], nodes.length[slot],
                                               !COMPACT && threadIdx.x < 3 ? grid[at] : 0.0,
                                               [&](uint32_t item, double (&v)[3]) {
                                                   values(item, v);
#pragma unroll
                                                   for (int c = 0; c < 3; ++c) v[c] = -v[c];
                                               });
            if (threadIdx.x < 3) grid[at] = acc;
            if (COMPACT && threadIdx.x == 0) density[node] = density[node] / samples_per_node;
        }
        return;
    }
    const uint32_t count = nodes.counters[0], stride = walk_blocks * blockDim.x;
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < count; slot += stride) {
        const uint32_t node = nodes.node[slot], length = nodes.length[slot];
        if (length > nodes.long_over) continue;
        const uint32_t* __restrict__ in = list + nodes.base[slot];
        const uint32_t at = COMPACT ? slot : node;
        double ax = 0.0, ay = 0.0, az = 0.0;
        if (!COMPACT) {
            ax = vx[node];
            ay = vy[node];
            az = vz[node];
        }
#pragma unroll 4
        for (uint32_t t = 0; t < length; ++t) {
            double v[3];
            values(in[t], v);
            ax -= v[0];
            ay -= v[1];
            az -= v[2];
        }
        vx[at] = ax;
        vy[at] = ay;
        vz[at] = az;
        if (COMPACT) density[node] = density[node] / samples_per_node;
    }
}

// rhs = -div V + point_weight screen h^-2 / 2 (capi.mojo:228-279) from V at the touched nodes: V is
// zero elsewhere, and a node away from all of them gets -0.0 + 0.0 = 0.0, as the dense kernel computes it.
// One thread per node, the slot map (4 bytes a node) read instead of three grids (24).
__global__ void __launch_bounds__(256) assemble_compact_kernel(const uint32_t* __restrict__ slot_of,
                                                               const double* __restrict__ vx,
                                                               const double* __restrict__ vy,
                                                               const double* __restrict__ vz,
                                                               const double* __restrict__ screen,
                                                               double* __restrict__ rhs, uint32_t n, int planes,
                                                               double point_weight, double target) {
    const uint32_t t = blockIdx.x * 256u + threadIdx.x, nn = n * n;
    if (t >= nn) return;
    const uint32_t y = t / n, x = t - y * n;
    const double h_inv = (double)(n - 1), h_inv2 = h_inv * h_inv, half_h = 0.5 * h_inv;
    const uint32_t z0 = blockIdx.y * planes, z1 = min(n, z0 + planes);
    uint32_t i = z0 * nn + t;
    uint32_t below = z0 ? slot_of[i - nn] : 0u, here = slot_of[i];
    for (uint32_t z = z0; z < z1; ++z, i += nn) {
        const uint32_t above = z + 1 < n ? slot_of[i + nn] : 0u;
        const uint32_t left = x ? slot_of[i - 1] : 0u, right = x + 1 < n ? slot_of[i + 1] : 0u;
        const uint32_t front = y ? slot_of[i - n] : 0u, back = y + 1 < n ? slot_of[i + n] : 0u;
        double value = 0.0;
        if (below | here | above | left | right | front | back) {
            auto get = [](const double* v, uint32_t slot) { return slot ? v[slot - 1] : 0.0; };
            double div = 0.0;
            if (x == 0) div += (get(vx, right) - get(vx, here)) * h_inv;
            else if (x == n - 1) div += (get(vx, here) - get(vx, left)) * h_inv;
            else div += (get(vx, right) - get(vx, left)) * half_h;
            if (y == 0) div += (get(vy, back) - get(vy, here)) * h_inv;
            else if (y == n - 1) div += (get(vy, here) - get(vy, front)) * h_inv;
            else div += (get(vy, back) - get(vy, front)) * half_h;
            if (z == 0) div += (get(vz, above) - get(vz, here)) * h_inv;
            else if (z == n - 1) div += (get(vz, here) - get(vz, below)) * h_inv;
            else div += (get(vz, above) - get(vz, below)) * half_h;
            value = -div + point_weight * (here ? screen[i] : 0.0) * h_inv2 * target;
        }
        rhs[i] = value;
        below = here;
        here = above;
    }
}

// ---- auxiliary attributes (upstream PoissonRecon's colour interpolation) --------
// Each sample's k attributes are splatted with its pass-1 weights w (the
// screening weights), per node in sample order: sum w a_c for c < k and, last,
// sum w.  One thread per (node, channel); DENSE: into planes of n^3, else rows of
// k + 1 per slot, from attributes in the points' sorted order (gather_attributes_kernel):
// the walk waits on its loads, and `order` would be one more in the chain of each.
__global__ void __launch_bounds__(256) gather_attributes_kernel(const double* __restrict__ attributes,
                                                                const uint32_t* __restrict__ order, int64_t count,
                                                                uint32_t channels, double* __restrict__ sorted) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)count * channels) return;
    const uint32_t place = (uint32_t)(i / channels), c = (uint32_t)(i - (uint64_t)place * channels);
    sorted[i] = attributes[(uint64_t)order[place] * channels + c];
}

template <bool DENSE>
__global__ void __launch_bounds__(256) attribute_sums_kernel(Nodes nodes, const uint32_t* __restrict__ list,
                                                             const Frac* __restrict__ frac,
                                                             const uint32_t* __restrict__ order,
                                                             const double* __restrict__ attributes, uint32_t channels,
                                                             int64_t plane, double* __restrict__ sums) {
    const uint64_t total = (uint64_t)nodes.counters[0] * (channels + 1), stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const uint32_t slot = (uint32_t)(i / (channels + 1)), c = (uint32_t)(i - (uint64_t)slot * (channels + 1));
        const uint32_t length = nodes.length[slot];
        const uint32_t* __restrict__ in = list + nodes.base[slot];
        double sum = 0.0;
#pragma unroll 4
        for (uint32_t t = 0; t < length; ++t) {
            const uint32_t item = in[t], place = item & ((1u << kPlaceBits) - 1u);
            const Frac f = load32(frac + place);
            const double w = corner_weight(f.x, f.y, f.z, f.weight, (int)(item >> kPlaceBits));
            if (f.weight != 0.0) sum += c < channels ? w * attributes[(int64_t)(DENSE ? order[place] : place) * channels + c] : w;
        }
        sums[DENSE ? c * plane + nodes.node[slot] : i] = sum;
    }
}

// sample_attributes_kernel over the slots' rows, one thread per (vertex, channel).
__global__ void __launch_bounds__(256) sample_slots_kernel(const double* __restrict__ vertices, int64_t count,
                                                           const double* __restrict__ map, int64_t n,
                                                           const uint32_t* __restrict__ slot_of,
                                                           const double* __restrict__ sums, uint32_t channels,
                                                           double* __restrict__ out) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)count * channels) return;
    const int64_t v = (int64_t)(i / channels);
    const uint32_t c = (uint32_t)(i - (uint64_t)v * channels);
    int64_t at[3];
    double f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) pass2_cell((vertices[3 * v + a] - map[a]) / map[3], n - 1, at[a], f[a]);
    double num = 0.0, den = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const double wz = (k & 4) ? f[2] : 1.0 - f[2];
        const double wy = (k & 2) ? f[1] : 1.0 - f[1];
        const double wx = (k & 1) ? f[0] : 1.0 - f[0];
        const uint32_t slot = slot_of[grid_index(at[0] + (k & 1), at[1] + ((k >> 1) & 1), at[2] + (k >> 2), n)];
        const double* row = sums + (uint64_t)(slot ? slot - 1 : 0) * (channels + 1);
        num += (slot ? row[c] : 0.0) * wx * wy * wz;
        den += (slot ? row[channels] : 0.0) * wx * wy * wz;
    }
    out[i] = den > 0.0 ? num / den : 0.0;
}

// Per vertex (world coordinates, mapped to the unit cube by `map` = (min x, y,
// z, width)): the ratio of the trilinear interpolants of sum w a_c and sum w
// over its cell (zero where no sample's weight reaches the cell).
__global__ void sample_attributes_kernel(const double* __restrict__ vertices, int64_t count,
                                         const double* __restrict__ map, int64_t n, const double* __restrict__ grids,
                                         int channels, double* __restrict__ out) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= count) return;
    const int64_t res = n - 1, plane = n * n * n;
    int64_t ix[3];
    double f[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double u = (vertices[3 * v + a] - map[a]) / map[3];
        pass2_cell(u, res, ix[a], f[a]);
    }
    double den = 0.0;
    for (int c = 0; c <= channels; ++c) {
        double num = 0.0;
        for (int dz = 0; dz < 2; ++dz) {
            const double wz = dz == 1 ? f[2] : 1.0 - f[2];
            for (int dy = 0; dy < 2; ++dy) {
                const double wy = dy == 1 ? f[1] : 1.0 - f[1];
                for (int dx = 0; dx < 2; ++dx) {
                    const double wx = dx == 1 ? f[0] : 1.0 - f[0];
                    num += grids[c * plane + grid_index(ix[0] + dx, ix[1] + dy, ix[2] + dz, n)] * wx * wy * wz;
                }
            }
        }
        if (c == channels) den = num;
        else out[v * channels + c] = num;
    }
    for (int c = 0; c < channels; ++c) out[v * channels + c] = den > 0.0 ? out[v * channels + c] / den : 0.0;
}

__global__ void store_count_kernel(const unsigned long long* __restrict__ src, int64_t* __restrict__ dst) {
    *dst = (int64_t)*src;
}

static int bit_width(uint64_t v) {
    int b = 0;
    while (v) {
        ++b;
        v >>= 1;
    }
    return b;
}


// What every splat shares: the points in cell order, the occupied cells, the touched nodes and
// their contributions.  The table of the cells (4 (n-1)^3 bytes) and the slot map (4 n^3) are dense.
struct Splat {
    int64_t count, n;
    uint32_t *keys, *keys_alt, *vals, *vals_alt, *rank, *heads, *cells, *table, *list;
    Frac* frac;
    Unit* unit;
    Nodes nodes;
    unsigned long long* accepted;

    // Lists longer than `over`, at most: a node has a point at most once.
    int64_t longs_at_most(uint32_t over = kLongOver) const { return count > over ? 8 * count / over : 0; }
    static int64_t node_capacity(int64_t count, int64_t n) { return std::min(8 * count, n * n * n); }

    // nodes_at_most: node_capacity(count, n), or 8 count where n is not known; table: carved unless given later
    void carve(Workspace& w, int64_t point_count, int64_t nodes_at_most, int64_t table_cells, int64_t map_nodes,
               bool units) {
        count = point_count;
        keys = w.take<uint32_t>(count);
        keys_alt = w.take<uint32_t>(count);
        vals = w.take<uint32_t>(count);
        vals_alt = w.take<uint32_t>(count);
        rank = w.take<uint32_t>(count);
        heads = w.take<uint32_t>(count + 1);
        cells = w.take<uint32_t>(1);
        list = w.take<uint32_t>(8 * count);
        frac = w.take<Frac>(count);
        unit = units ? w.take<Unit>(count) : nullptr;
        nodes.node = w.take<uint32_t>(nodes_at_most);
        nodes.base = w.take<uint32_t>(nodes_at_most);
        nodes.length = w.take<uint32_t>(nodes_at_most);
        nodes.counters = w.take<uint32_t>(4);
        nodes.units = w.take<uint2>(8 * count / kUnit + longs_at_most());
        nodes.longs = w.take<uint32_t>(longs_at_most());
        accepted = w.take<unsigned long long>(1);
        table = table_cells ? w.take<uint32_t>(table_cells) : nullptr;
        nodes.slot_of = map_nodes ? w.take<uint32_t>(map_nodes) : nullptr;
    }

    static void carve_scratch(Workspace& w, int64_t count) {
        radix_carve<uint32_t>(w, count);
        scan_carve<uint32_t>(w, count);
    }

    Cells geometry() const {
        return Cells{(uint32_t)n, (uint32_t)(n - 1), FastDiv((uint32_t)(n - 1)), FastDiv((uint32_t)n), table, heads};
    }

    // Up to the touched nodes; keys and vals are the sorted ones afterwards.
    int group(const double* points, const double* normals, int64_t side, int confidence, Workspace& w, cudaStream_t s) {
        n = side;
        nodes.long_over = long_over_of(n);
        const int64_t c = n - 1;
        const unsigned blocks = blocks_for(count, 256);
        PB_CHECK_CUDA(cudaMemsetAsync(accepted, 0, sizeof(unsigned long long), s), "splat accepted");
        PB_CHECK_CUDA(cudaMemsetAsync(nodes.counters, 0, 4 * sizeof(uint32_t), s), "splat counters");
        PB_CHECK_CUDA(cudaMemsetAsync(table, 0, (size_t)(c * c * c) * sizeof(uint32_t), s), "splat table");
        if (nodes.slot_of)
            PB_CHECK_CUDA(cudaMemsetAsync(nodes.slot_of, 0, (size_t)(n * n * n) * sizeof(uint32_t), s), "splat map");
        cell_keys_kernel<<<blocks, 256, 0, s>>>(points, normals, count, n, keys, vals, accepted);
        PB_CHECK_LAUNCH("cell_keys_kernel");
        bool in_alt = false;
        PB_TRY(radix_sort_pairs<uint32_t>(keys, vals, keys_alt, vals_alt, count, bit_width((uint64_t)(c * c * c - 1)),
                                          &in_alt, w, s));
        if (in_alt) {
            std::swap(keys, keys_alt);
            std::swap(vals, vals_alt);
        }
        gather_points_kernel<<<blocks, 256, 0, s>>>(points, normals, count, n, confidence, keys, vals, frac, unit, rank);
        PB_CHECK_LAUNCH("gather_points_kernel");
        PB_TRY(exclusive_scan<uint32_t>(rank, rank, count, cells, w, s));
        cell_table_kernel<<<blocks, 256, 0, s>>>(keys, rank, count, cells, heads, table);
        PB_CHECK_LAUNCH("cell_table_kernel");
        touched_nodes_kernel<<<(unsigned)std::min<int64_t>(blocks_for(count, 128), 32 * kSMs), 128, 0, s>>>(
            geometry(), keys, cells, nodes);
        PB_CHECK_LAUNCH("touched_nodes_kernel");
        return PB_OK;
    }

    unsigned node_blocks(int per_node = 1) const {
        return (unsigned)std::min<int64_t>(blocks_for(node_capacity(count, n) * per_node, 256), 16 * kSMs);
    }

    // Blocks for the long lists (four resident ones per SM) and for their parts; none where no list can be long.
    unsigned long_blocks() const { return (unsigned)std::min<int64_t>(longs_at_most(nodes.long_over), 4 * kSMs); }
    unsigned unit_blocks() const {
        return long_blocks() ? (unsigned)std::min<int64_t>(8 * count / kUnit + 1, 16 * kSMs) : 0;
    }

    // The nodes' contributions in order; pass 1 into dense grids unless they are null.
    int merge(double* density, double* screen, cudaStream_t s) const {
        const unsigned ranks = unit_blocks(), blocks = ranks + node_blocks();
        (density ? merge_kernel<true> : merge_kernel<false>)<<<blocks, 256, 0, s>>>(geometry(), nodes, vals, frac, list,
                                                                                   density, screen, ranks);
        PB_CHECK_LAUNCH("merge_kernel");
        if (density && long_blocks()) {
            long_sums_kernel<<<long_blocks(), 256, 0, s>>>(nodes, list, frac, density, screen);
            PB_CHECK_LAUNCH("long_sums_kernel");
        }
        return PB_OK;
    }

    // Pass 2 into dense grids, or (compact) into slots, dividing the density.
    int pass2(double* density, double samples_per_node, double* vx, double* vy, double* vz, bool compact,
              cudaStream_t s) const {
        density_factor_kernel<<<blocks_for(count, 256), 256, 0, s>>>(count, n, keys, frac, samples_per_node, density,
                                                                     unit);
        PB_CHECK_LAUNCH("density_factor_kernel");
        (compact ? vector_kernel<true> : vector_kernel<false>)<<<long_blocks() + node_blocks(), 256, 0, s>>>(
            nodes, list, frac, unit, (double)(n - 1), vx, vy, vz, density, samples_per_node, long_blocks());
        PB_CHECK_LAUNCH("vector_kernel");
        return PB_OK;
    }

    int store_accepted(int64_t* out, cudaStream_t s) const {
        store_count_kernel<<<1, 1, 0, s>>>(accepted, out);
        PB_CHECK_LAUNCH("store_count_kernel");
        return PB_OK;
    }
};

static int64_t cubed(int64_t v) { return v * v * v; }

static int check_splat(const char* what, const double* points, const double* normals, int64_t point_count, int64_t n) {
    if (n < 2) return fail(PB_ERR_INVALID, "%s: n must be >= 2", what);
    if (cubed(n) >= (int64_t)0x7FFFFFFF) return fail(PB_ERR_INVALID, "%s: n^3 must be < 2^31", what);
    if (point_count < 0 || point_count * 8 >= (int64_t)0xFFFFFFFFll)
        return fail(PB_ERR_INVALID, "%s: point_count must be in [0, 2^29)", what);
    if (point_count && (!points || !normals)) return fail(PB_ERR_INVALID, "%s: null points/normals", what);
    return PB_OK;
}

// V at the touched nodes for pb_splat_assemble_f64.
struct CompactVectors {
    double *x, *y, *z;
    void carve(Workspace& w, int64_t nodes) {
        x = w.take<double>(nodes);
        y = w.take<double>(nodes);
        z = w.take<double>(nodes);
    }
};

static size_t splat_ws_bytes(int64_t count, int64_t n, bool assemble) {
    return measure([&](Workspace& w) {
        Splat o;
        const int64_t cap = Splat::node_capacity(count, n);
        o.carve(w, count, cap, cubed(n - 1), assemble ? cubed(n) : 0, true);
        CompactVectors v;
        if (assemble) v.carve(w, cap);
        Splat::carve_scratch(w, count);
    });
}

static int64_t side_for_size(int64_t n) { return n < 2 ? 2 : n > 1290 ? 1290 : n; }

}  // namespace pb

using namespace pb;

extern "C" size_t pb_splat_workspace_size(int64_t point_count, int64_t n) {
    return splat_ws_bytes(point_count < 1 ? 1 : point_count, side_for_size(n), false);
}

extern "C" int pb_splat_f64(const double* points, const double* normals, int64_t point_count, int64_t n,
                            int64_t confidence, double* density, double* vx, double* vy, double* vz, double* screen,
                            double samples_per_node, int64_t* accepted, void* workspace, size_t workspace_bytes,
                            void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    PB_TRY(check_splat("splat", points, normals, point_count, n));
    if (!accepted || !density || !vx || !vy || !vz || !screen) return fail(PB_ERR_INVALID, "splat: null buffer");
    if (point_count == 0) {
        PB_CHECK_CUDA(cudaMemsetAsync(accepted, 0, sizeof(int64_t), s), "splat accepted");
        return PB_OK;
    }
    const size_t need = splat_ws_bytes(point_count, n, false);
    if (!workspace || workspace_bytes < need) return fail(PB_ERR_WORKSPACE, "splat: workspace needs %zu bytes", need);
    Workspace w(workspace, workspace_bytes);
    Splat o;
    o.carve(w, point_count, Splat::node_capacity(point_count, n), cubed(n - 1), 0, true);
    PB_TRY(o.group(points, normals, n, (int)confidence, w, s));
    PB_TRY(o.merge(density, screen, s));
    PB_TRY(o.pass2(density, samples_per_node, vx, vy, vz, false, s));
    return o.store_accepted(accepted, s);
}

extern "C" size_t pb_splat_assemble_workspace_size(int64_t point_count, int64_t n) {
    return splat_ws_bytes(point_count < 1 ? 1 : point_count, side_for_size(n), true);
}

// Splat and assembly from points to the solver's grids (core.py:228-265): density (divided by
// samples_per_node), screen and rhs, all n^3 and overwritten; the same bits as zeroed grids through
// pb_splat_f64, pb_divide_f64 and pb_assemble_f64.  The vector field exists only at the touched nodes.
extern "C" int pb_splat_assemble_f64(const double* points, const double* normals, int64_t point_count, int64_t n,
                                     int64_t confidence, double samples_per_node, double point_weight,
                                     double target_value, double* density, double* screen, double* rhs,
                                     int64_t* accepted, void* workspace, size_t workspace_bytes, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    PB_TRY(check_splat("splat assemble", points, normals, point_count, n));
    if (!accepted || !density || !screen || !rhs) return fail(PB_ERR_INVALID, "splat assemble: null buffer");
    const size_t grid = (size_t)cubed(n) * sizeof(double);
    PB_CHECK_CUDA(cudaMemsetAsync(density, 0, grid, s), "splat assemble density");
    PB_CHECK_CUDA(cudaMemsetAsync(screen, 0, grid, s), "splat assemble screen");
    if (point_count == 0) {
        PB_CHECK_CUDA(cudaMemsetAsync(rhs, 0, grid, s), "splat assemble rhs");
        PB_CHECK_CUDA(cudaMemsetAsync(accepted, 0, sizeof(int64_t), s), "splat assemble accepted");
        return PB_OK;
    }
    const size_t need = splat_ws_bytes(point_count, n, true);
    if (!workspace || workspace_bytes < need)
        return fail(PB_ERR_WORKSPACE, "splat assemble: workspace needs %zu bytes", need);
    Workspace w(workspace, workspace_bytes);
    const int64_t cap = Splat::node_capacity(point_count, n);
    Splat o;
    o.carve(w, point_count, cap, cubed(n - 1), cubed(n), true);
    CompactVectors v;
    v.carve(w, cap);
    PB_TRY(o.group(points, normals, n, (int)confidence, w, s));
    PB_TRY(o.merge(density, screen, s));
    PB_TRY(o.pass2(density, samples_per_node, v.x, v.y, v.z, true, s));
    const int planes = n >= 129 ? 8 : 2;
    assemble_compact_kernel<<<dim3(blocks_for(n * n, 256), (unsigned)((n + planes - 1) / planes)), 256, 0, s>>>(
        o.nodes.slot_of, v.x, v.y, v.z, screen, rhs, (uint32_t)n, planes, point_weight, target_value);
    PB_CHECK_LAUNCH("assemble_compact_kernel");
    return o.store_accepted(accepted, s);
}

namespace pb {

static size_t attr_ws_bytes(int64_t count) {
    return measure([&](Workspace& w) {
        Splat o;
        o.carve(w, count, 8 * count, 0, 0, false);
        Splat::carve_scratch(w, count);
    });
}

static size_t interpolate_ws_bytes(int64_t count, int64_t n, int64_t channels) {
    return measure([&](Workspace& w) {
        Splat o;
        const int64_t cap = Splat::node_capacity(count, n);
        o.carve(w, count, cap, cubed(n - 1), cubed(n), false);
        w.take<double>(cap * (channels + 1));
        w.take<double>(count * channels);
        Splat::carve_scratch(w, count);
    });
}

}  // namespace pb

extern "C" size_t pb_splat_attributes_workspace_size(int64_t point_count) {
    return attr_ws_bytes(point_count < 1 ? 1 : point_count);
}

// Auxiliary attributes of unit-cube samples (points, normals as for
// pb_splat_f64; attributes: point_count x channels, row-major): grids (channels
// + 1 planes of n^3, overwritten) get sum w a_c per node and, in the last
// plane, sum w, with w the samples' pass-1 weights, summed in sample order.
extern "C" int pb_splat_attributes_f64(const double* points, const double* normals, int64_t point_count, int64_t n,
                                       int64_t confidence, const double* attributes, int64_t channels,
                                       double* grids, void* workspace, size_t workspace_bytes, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    if (n < 2 || n * n * n >= (int64_t)0x7FFFFFFF) return fail(PB_ERR_INVALID, "splat attributes: bad n");
    if (point_count < 0 || point_count * 8 >= (int64_t)0xFFFFFFFFll || channels < 1 || channels > 64 || !grids)
        return fail(PB_ERR_INVALID, "splat attributes: bad sizes");
    const size_t bytes = sizeof(double) * (size_t)(channels + 1) * (size_t)cubed(n);
    if (point_count == 0) {
        PB_CHECK_CUDA(cudaMemsetAsync(grids, 0, bytes, s), "splat attributes zero");
        return PB_OK;
    }
    if (!points || !normals || !attributes) return fail(PB_ERR_INVALID, "splat attributes: null input");
    const size_t need = attr_ws_bytes(point_count);
    if (!workspace || workspace_bytes < need)
        return fail(PB_ERR_WORKSPACE, "splat attributes: workspace needs %zu bytes", need);
    Workspace w(workspace, workspace_bytes);
    Splat o;
    o.carve(w, point_count, 8 * point_count, 0, 0, false);
    o.table = (uint32_t*)grids;  // the cells' table until the nodes' contributions are listed
    PB_TRY(o.group(points, normals, n, (int)confidence, w, s));
    PB_TRY(o.merge(nullptr, nullptr, s));
    PB_CHECK_CUDA(cudaMemsetAsync(grids, 0, bytes, s), "splat attributes zero");
    attribute_sums_kernel<true><<<o.node_blocks((int)channels + 1), 256, 0, s>>>(
        o.nodes, o.list, o.frac, o.vals, attributes, (uint32_t)channels, cubed(n), grids);
    PB_CHECK_LAUNCH("attribute_sums_kernel");
    return PB_OK;
}

// Attribute values at mesh vertices (world coordinates; map = the (min x, y, z,
// width) that took the samples to the unit cube): out (vertex_count x
// channels) from the grids of pb_splat_attributes_f64.
extern "C" int pb_sample_attributes_f64(const double* vertices, int64_t vertex_count, const double* map, int64_t n,
                                        const double* grids, int64_t channels, double* out, void* stream) {
    if (n < 2 || vertex_count < 0 || channels < 1 || channels > 64 || !map || !grids ||
        (vertex_count && (!vertices || !out)))
        return fail(PB_ERR_INVALID, "sample attributes: bad args");
    if (!vertex_count) return PB_OK;
    sample_attributes_kernel<<<blocks_for(vertex_count, 256), 256, 0, (cudaStream_t)stream>>>(
        vertices, vertex_count, map, n, grids, (int)channels, out);
    PB_CHECK_LAUNCH("sample_attributes_kernel");
    return PB_OK;
}

extern "C" size_t pb_interpolate_attributes_workspace_size(int64_t point_count, int64_t n, int64_t channels) {
    return interpolate_ws_bytes(point_count < 1 ? 1 : point_count, side_for_size(n),
                                channels < 1 ? 1 : channels > 64 ? 64 : channels);
}

// pb_splat_attributes_f64 and pb_sample_attributes_f64 in one call, the sums kept only at the
// touched nodes (rows of channels + 1 instead of as many planes of n^3).  Same bits.
extern "C" int pb_interpolate_attributes_f64(const double* points, const double* normals, int64_t point_count,
                                             int64_t n, int64_t confidence, const double* attributes, int64_t channels,
                                             const double* vertices, int64_t vertex_count, const double* map,
                                             double* out, void* workspace, size_t workspace_bytes, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    PB_TRY(check_splat("interpolate attributes", points, normals, point_count, n));
    if (channels < 1 || channels > 64 || vertex_count < 0 || (point_count && !attributes) ||
        (vertex_count && (!vertices || !map || !out)))
        return fail(PB_ERR_INVALID, "interpolate attributes: bad args");
    if (!vertex_count) return PB_OK;
    if (!point_count) {
        PB_CHECK_CUDA(cudaMemsetAsync(out, 0, (size_t)vertex_count * channels * sizeof(double), s), "interpolate zero");
        return PB_OK;
    }
    const size_t need = interpolate_ws_bytes(point_count, n, channels);
    if (!workspace || workspace_bytes < need)
        return fail(PB_ERR_WORKSPACE, "interpolate attributes: workspace needs %zu bytes", need);
    Workspace w(workspace, workspace_bytes);
    const int64_t cap = Splat::node_capacity(point_count, n);
    Splat o;
    o.carve(w, point_count, cap, cubed(n - 1), cubed(n), false);
    double* sums = w.take<double>(cap * (channels + 1));
    double* sorted = w.take<double>(point_count * channels);
    PB_TRY(o.group(points, normals, n, (int)confidence, w, s));
    PB_TRY(o.merge(nullptr, nullptr, s));
    gather_attributes_kernel<<<blocks_for(point_count * channels, 256), 256, 0, s>>>(attributes, o.vals, point_count,
                                                                                    (uint32_t)channels, sorted);
    PB_CHECK_LAUNCH("gather_attributes_kernel");
    attribute_sums_kernel<false><<<o.node_blocks((int)channels + 1), 256, 0, s>>>(
        o.nodes, o.list, o.frac, nullptr, sorted, (uint32_t)channels, 0, sums);
    PB_CHECK_LAUNCH("attribute_sums_kernel");
    sample_slots_kernel<<<blocks_for(vertex_count * channels, 256), 256, 0, s>>>(
        vertices, vertex_count, map, n, o.nodes.slot_of, sums, (uint32_t)channels, out);
    PB_CHECK_LAUNCH("sample_slots_kernel");
    return PB_OK;
}
