// Two-pass dual contouring (surface nets), order-preserving.
//
// Reference: src/capi.mojo:798-1129.  The reference numbers active cells
// serially in z,y,x order and emits quads in three serial sweeps (x-edges,
// y-edges, z-edges, each in z,y,x order).  Here both orders come from stream
// compaction: (1) per-tile counts, (2) an exclusive scan of the tile counts,
// (3) each tile recomputes its flags, scans them within the block and writes
// element i at (tile offset + rank).  Ids, vertex order and face order are
// therefore identical to the serial reference; vertex coordinates are exact
// restatements (compiled with -fmad=false).
#include <algorithm>

#include "scan.cuh"

namespace pb {

constexpr int kDualThreads = 256;
constexpr int kDualItems = 8;
constexpr int kDualTile = kDualThreads * kDualItems;

struct IsoArg {
    double value;
    const double* ptr;
    __device__ __forceinline__ double get() const { return ptr ? *ptr : value; }
};

__device__ __forceinline__ bool cell_active(const double* __restrict__ f, int64_t x, int64_t y, int64_t z, int64_t n,
                                            double iso) {
    const int64_t i0 = (z * n + y) * n + x;
    const int64_t sy = n, sz = n * n;
    int below = (f[i0] < iso) + (f[i0 + 1] < iso) + (f[i0 + sy] < iso) + (f[i0 + sy + 1] < iso) +
                (f[i0 + sz] < iso) + (f[i0 + sz + 1] < iso) + (f[i0 + sz + sy] < iso) + (f[i0 + sz + sy + 1] < iso);
    return below != 0 && below != 8;
}

__global__ void __launch_bounds__(kDualThreads) cell_count_kernel(const double* __restrict__ field, int64_t n,
                                                                  IsoArg iso_arg, int64_t* __restrict__ tile_counts) {
    __shared__ int64_t warp_sums[32];
    const int64_t cells = n - 1;
    const int64_t total = cells * cells * cells;
    const double iso = iso_arg.get();
    const int64_t base = (int64_t)blockIdx.x * kDualTile + (int64_t)threadIdx.x * kDualItems;
    int64_t c = 0;
#pragma unroll
    for (int k = 0; k < kDualItems; ++k) {
        const int64_t i = base + k;
        if (i < total) {
            const int64_t x = i % cells, y = (i / cells) % cells, z = i / (cells * cells);
            c += cell_active(field, x, y, z, n, iso);
        }
    }
    int64_t t;
    block_exclusive_scan<int64_t>(c, warp_sums, t);
    if (threadIdx.x == 0) tile_counts[blockIdx.x] = t;
}

// capi.mojo:812-836
__device__ __forceinline__ int edge_root(double v0, double v1, double iso, double x0, double y0, double z0, double x1,
                                         double y1, double z1, double& sx, double& sy, double& sz) {
    if ((v0 < iso) == (v1 < iso)) return 0;
    double t = (iso - v0) / (v1 - v0);
    t = t > 0.0 ? t : 0.0;
    t = t < 1.0 ? t : 1.0;
    sx = sx + x0 + (x1 - x0) * t;
    sy = sy + y0 + (y1 - y0) * t;
    sz = sz + z0 + (z1 - z0) * t;
    return 1;
}

// Vertex of active cell (x, y, z): the mean of its edge roots (capi.mojo:964-1033),
// and the mean density of its corners.
__device__ __forceinline__ void cell_vertex(const double* __restrict__ field, const double* __restrict__ density,
                                            int64_t n, int64_t x, int64_t y, int64_t z, double iso, double cells_d,
                                            double* __restrict__ out, double* __restrict__ dens) {
    double v[8];
#pragma unroll
    for (int corner = 0; corner < 8; ++corner)
        v[corner] = field[grid_index(x + (corner & 1), y + ((corner >> 1) & 1), z + ((corner >> 2) & 1), n)];
    double sx = 0.0, sy = 0.0, sz = 0.0;
    int roots = 0;
    // x-edges, y-edges, z-edges; within each, (a, b) in row-major order (capi.mojo:968-1023).
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int c0 = 2 * a + 4 * b;
            roots += edge_root(v[c0], v[c0 + 1], iso, 0.0, (double)a, (double)b, 1.0, (double)a, (double)b, sx, sy, sz);
        }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int c0 = a + 4 * b;
            roots += edge_root(v[c0], v[c0 + 2], iso, (double)a, 0.0, (double)b, (double)a, 1.0, (double)b, sx, sy, sz);
        }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int c0 = a + 2 * b;
            roots += edge_root(v[c0], v[c0 + 4], iso, (double)a, (double)b, 0.0, (double)a, (double)b, 1.0, sx, sy, sz);
        }
    const double inv_roots = 1.0 / (double)roots;
    out[0] = ((double)x + sx * inv_roots) / cells_d;
    out[1] = ((double)y + sy * inv_roots) / cells_d;
    out[2] = ((double)z + sz * inv_roots) / cells_d;
    double dsum = 0.0;
#pragma unroll
    for (int corner = 0; corner < 8; ++corner)
        dsum += density[grid_index(x + (corner & 1), y + ((corner >> 1) & 1), z + ((corner >> 2) & 1), n)];
    *dens = dsum * 0.125;
}

__global__ void __launch_bounds__(kDualThreads) vertex_emit_kernel(const double* __restrict__ field,
                                                                   const double* __restrict__ density, int64_t n,
                                                                   IsoArg iso_arg,
                                                                   const int64_t* __restrict__ tile_offsets,
                                                                   int64_t capacity, int64_t* __restrict__ cell_map,
                                                                   double* __restrict__ vertices,
                                                                   double* __restrict__ vertex_density) {
    __shared__ int64_t warp_sums[32];
    const int64_t cells = n - 1;
    const int64_t total = cells * cells * cells;
    const double iso = iso_arg.get();
    const int64_t base = (int64_t)blockIdx.x * kDualTile + (int64_t)threadIdx.x * kDualItems;
    unsigned active = 0;
    int64_t c = 0;
#pragma unroll
    for (int k = 0; k < kDualItems; ++k) {
        const int64_t i = base + k;
        if (i < total) {
            const int64_t x = i % cells, y = (i / cells) % cells, z = i / (cells * cells);
            if (cell_active(field, x, y, z, n, iso)) {
                active |= 1u << k;
                ++c;
            }
        }
    }
    int64_t t;
    int64_t id = tile_offsets[blockIdx.x] + block_exclusive_scan<int64_t>(c, warp_sums, t);
    const double cells_d = (double)cells;
    for (int k = 0; k < kDualItems; ++k) {
        const int64_t i = base + k;
        if (i >= total) break;
        if (!(active & (1u << k))) {
            cell_map[i] = -1;
            continue;
        }
        if (id >= capacity) {  // capi.mojo:961-963: past capacity, the cell keeps 0
            cell_map[i] = 0;
            ++id;
            continue;
        }
        const int64_t x = i % cells, y = (i / cells) % cells, z = i / (cells * cells);
        cell_vertex(field, density, n, x, y, z, iso, cells_d, vertices + 3 * id, vertex_density + id);
        cell_map[i] = id;
        ++id;
    }
}

// Edge e of the three sweeps (capi.mojo:1090-1128).  Each sweep has
// cells*(cells-1)^2 edges; returns the quad's four cells (cell indices) and
// whether the edge changes sign, with v0 < iso for the orientation.
__device__ __forceinline__ bool edge_quad(const double* __restrict__ f, const int64_t* __restrict__ cm, int64_t n,
                                          double iso, int64_t e, int64_t per_sweep, int64_t q[4], bool& reverse) {
    const int64_t cells = n - 1;
    const int sweep = (int)(e / per_sweep);
    const int64_t local = e - (int64_t)sweep * per_sweep;
    int64_t x, y, z;
    const int64_t cm1 = cells - 1;
    double v0, v1;
    if (sweep == 0) {  // z in [1,cells), y in [1,cells), x in [0,cells)
        x = local % cells;
        y = 1 + (local / cells) % cm1;
        z = 1 + local / (cells * cm1);
        v0 = f[grid_index(x, y, z, n)];
        v1 = f[grid_index(x + 1, y, z, n)];
    } else if (sweep == 1) {  // z in [1,cells), y in [0,cells), x in [1,cells)
        x = 1 + local % cm1;
        y = (local / cm1) % cells;
        z = 1 + local / (cm1 * cells);
        v0 = f[grid_index(x, y, z, n)];
        v1 = f[grid_index(x, y + 1, z, n)];
    } else {  // z in [0,cells), y in [1,cells), x in [1,cells)
        x = 1 + local % cm1;
        y = 1 + (local / cm1) % cm1;
        z = local / (cm1 * cm1);
        v0 = f[grid_index(x, y, z, n)];
        v1 = f[grid_index(x, y, z + 1, n)];
    }
    if ((v0 < iso) == (v1 < iso)) return false;
    reverse = v0 < iso;
    if (sweep == 0) {
        q[0] = grid_index(x, y - 1, z - 1, cells);
        q[1] = grid_index(x, y, z - 1, cells);
        q[2] = grid_index(x, y, z, cells);
        q[3] = grid_index(x, y - 1, z, cells);
    } else if (sweep == 1) {
        q[0] = grid_index(x - 1, y, z - 1, cells);
        q[1] = grid_index(x - 1, y, z, cells);
        q[2] = grid_index(x, y, z, cells);
        q[3] = grid_index(x, y, z - 1, cells);
    } else {
        q[0] = grid_index(x - 1, y - 1, z, cells);
        q[1] = grid_index(x, y - 1, z, cells);
        q[2] = grid_index(x, y, z, cells);
        q[3] = grid_index(x - 1, y, z, cells);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        q[k] = cm[q[k]];
        if (q[k] < 0) return false;  // capi.mojo:1055-1056
    }
    return true;
}

__global__ void __launch_bounds__(kDualThreads) face_count_kernel(const double* __restrict__ field,
                                                                  const int64_t* __restrict__ cm, int64_t n,
                                                                  IsoArg iso_arg, int64_t per_sweep,
                                                                  int64_t* __restrict__ tile_counts) {
    __shared__ int64_t warp_sums[32];
    const int64_t total = 3 * per_sweep;
    const double iso = iso_arg.get();
    const int64_t base = (int64_t)blockIdx.x * kDualTile + (int64_t)threadIdx.x * kDualItems;
    int64_t c = 0;
    for (int k = 0; k < kDualItems; ++k) {
        const int64_t e = base + k;
        if (e >= total) break;
        int64_t q[4];
        bool rev;
        c += edge_quad(field, cm, n, iso, e, per_sweep, q, rev);
    }
    int64_t t;
    block_exclusive_scan<int64_t>(c, warp_sums, t);
    if (threadIdx.x == 0) tile_counts[blockIdx.x] = t;
}

__global__ void __launch_bounds__(kDualThreads) face_emit_kernel(const double* __restrict__ field,
                                                                 const int64_t* __restrict__ cm, int64_t n,
                                                                 IsoArg iso_arg, int64_t per_sweep,
                                                                 const int64_t* __restrict__ tile_offsets,
                                                                 int64_t capacity, int64_t* __restrict__ faces) {
    __shared__ int64_t warp_sums[32];
    const int64_t total = 3 * per_sweep;
    const double iso = iso_arg.get();
    const int64_t base = (int64_t)blockIdx.x * kDualTile + (int64_t)threadIdx.x * kDualItems;
    int64_t q[kDualItems][4];
    unsigned emit = 0, rev = 0;
    int64_t c = 0;
#pragma unroll
    for (int k = 0; k < kDualItems; ++k) {
        const int64_t e = base + k;
        bool r = false;
        if (e < total && edge_quad(field, cm, n, iso, e, per_sweep, q[k], r)) {
            emit |= 1u << k;
            if (r) rev |= 1u << k;
            ++c;
        }
    }
    int64_t t;
    int64_t quad = tile_offsets[blockIdx.x] + block_exclusive_scan<int64_t>(c, warp_sums, t);
#pragma unroll
    for (int k = 0; k < kDualItems; ++k) {
        if (!(emit & (1u << k))) continue;
        const int64_t fc = 2 * quad;
        if (fc + 2 <= capacity) {  // capi.mojo:1057-1071
            int64_t* out = faces + 3 * fc;
            const int64_t a = q[k][0], b = q[k][1], cc = q[k][2], d = q[k][3];
            if (rev & (1u << k)) {
                out[0] = a; out[1] = d; out[2] = cc; out[3] = a; out[4] = cc; out[5] = b;
            } else {
                out[0] = a; out[1] = b; out[2] = cc; out[3] = a; out[4] = cc; out[5] = d;
            }
        }
        ++quad;
    }
}

__global__ void double_count_kernel(int64_t* __restrict__ count) { *count = 2 * *count; }

static int64_t tiles_of(int64_t items) { return (items + kDualTile - 1) / kDualTile; }

static size_t dual_ws_bytes(int64_t n) {
    const int64_t cells = n - 1;
    const int64_t vt = tiles_of(cells * cells * cells);
    const int64_t ft = tiles_of(3 * cells * (cells - 1) * (cells - 1));
    const int64_t tiles = vt > ft ? vt : ft;
    return measure([&](Workspace& w) {
        w.take<int64_t>(tiles);
        scan_carve<int64_t>(w, tiles);
    });
}

static int dual_vertices(const double* field, const double* density, int64_t n, IsoArg iso, int64_t* cell_map,
                         double* vertices, double* vertex_density, int64_t capacity, int64_t* count, void* workspace,
                         size_t workspace_bytes, cudaStream_t s) {
    if (n < 2 || n > 4097) return fail(PB_ERR_INVALID, "dual vertices: n must be in [2, 4097]");
    if (!field || !count) return fail(PB_ERR_INVALID, "dual vertices: null buffer");
    if (capacity > 0 && (!density || !cell_map || !vertices || !vertex_density))
        return fail(PB_ERR_INVALID, "dual vertices: null output buffer");
    const size_t need = dual_ws_bytes(n);
    if (!workspace || workspace_bytes < need) return fail(PB_ERR_WORKSPACE, "dual: workspace needs %zu bytes", need);
    Workspace w(workspace, workspace_bytes);
    const int64_t cells = n - 1;
    const int64_t total = cells * cells * cells;
    const int64_t tiles = tiles_of(total);
    int64_t* tile_counts = w.take<int64_t>(tiles);
    cell_count_kernel<<<(unsigned)tiles, kDualThreads, 0, s>>>(field, n, iso, tile_counts);
    PB_CHECK_LAUNCH("cell_count_kernel");
    PB_TRY(exclusive_scan<int64_t>(tile_counts, tile_counts, tiles, count, w, s));
    if (capacity > 0) {
        vertex_emit_kernel<<<(unsigned)tiles, kDualThreads, 0, s>>>(field, density, n, iso, tile_counts, capacity,
                                                                    cell_map, vertices, vertex_density);
        PB_CHECK_LAUNCH("vertex_emit_kernel");
    }
    return PB_OK;
}

static int dual_faces(const double* field, int64_t n, IsoArg iso, const int64_t* cell_map, int64_t* faces,
                      int64_t capacity, int64_t* count, void* workspace, size_t workspace_bytes, cudaStream_t s) {
    if (n < 2 || n > 4097) return fail(PB_ERR_INVALID, "dual faces: n must be in [2, 4097]");
    if (!field || !count || !cell_map) return fail(PB_ERR_INVALID, "dual faces: null buffer");
    if (capacity > 0 && !faces) return fail(PB_ERR_INVALID, "dual faces: null faces");
    const size_t need = dual_ws_bytes(n);
    if (!workspace || workspace_bytes < need) return fail(PB_ERR_WORKSPACE, "dual: workspace needs %zu bytes", need);
    const int64_t cells = n - 1;
    const int64_t per_sweep = cells * (cells - 1) * (cells - 1);
    if (per_sweep == 0) {
        PB_CHECK_CUDA(cudaMemsetAsync(count, 0, sizeof(int64_t), s), "dual faces count");
        return PB_OK;
    }
    Workspace w(workspace, workspace_bytes);
    const int64_t tiles = tiles_of(3 * per_sweep);
    int64_t* tile_counts = w.take<int64_t>(tiles);
    face_count_kernel<<<(unsigned)tiles, kDualThreads, 0, s>>>(field, cell_map, n, iso, per_sweep, tile_counts);
    PB_CHECK_LAUNCH("face_count_kernel");
    PB_TRY(exclusive_scan<int64_t>(tile_counts, tile_counts, tiles, count, w, s));
    if (capacity > 0) {
        face_emit_kernel<<<(unsigned)tiles, kDualThreads, 0, s>>>(field, cell_map, n, iso, per_sweep, tile_counts,
                                                                  capacity, faces);
        PB_CHECK_LAUNCH("face_emit_kernel");
    }
    double_count_kernel<<<1, 1, 0, s>>>(count);  // two triangles per quad
    PB_CHECK_LAUNCH("double_count_kernel");
    return PB_OK;
}


// ---- extraction for reconstruct(): sign bits and rank structures ----------------
// Same output, order and arithmetic as the two-pass kernels above.  One pass over
// the field leaves one bit per node (field < iso), rows (y, z) starting on a 32-bit
// word of their own.  The 32 cells, and the 32 edges of each sweep, that start in a
// word of row (y, z) then follow from the words of rows (y .. y + 1, z .. z + 1) and
// the same words shifted by one node, all 32 at once: four words of active cells and
// sign-changing x-, y- and z-edges per row word, in four segments that a prefix sum
// of popcounts ranks in the reference's order (word order is z, y, x order).  The
// emission writes every active item's place into the first slot of its own output,
// one thread per word, and then runs one thread per vertex and per quad; vertex ids
// are ranks in the cell words.  Only active cells read field and density values.
// Sides up to 1025.
// Against one ballot per 32 cells or edges and one thread per word emitting its
// items, all kernels together at 230^3 with 677 K vertices: 340 -> 115 us on B200
// (sign rows 23, words and ranks 12, places 24, vertices 34, quads 23).
namespace fast {

constexpr int kT = 256;
constexpr int64_t kMaxSide = 1025;
constexpr int kTileWords = kScanThreads * kScanItems;  // words per block of the popcount scan

__device__ __forceinline__ uint32_t lanes_below(uint32_t word, uint32_t b) { return __popc(word & ((1u << b) - 1u)); }

// Row words of the sign bits (n + 31) / 32 and of the cells' (c + 31) / 32, c = n - 1.
struct Rows {
    uint32_t n, c, sign_words, words, segment;  // segment: c^2 words of one kind, rounded up to whole scan tiles
    FastDiv by_words, by_c;
    __host__ explicit Rows(int64_t side)
        : n((uint32_t)side), c(n - 1), sign_words((n + 31) / 32), words((c + 31) / 32),
          segment((c * c * words + kTileWords - 1) / kTileWords * kTileWords), by_words(words), by_c(c) {}
};

// bits: bit x & 31 of word x >> 5 of row (y, z) = (field < iso), one warp per row;
// *bad |= 1 (bad may be null) if a value is not finite.
__global__ void __launch_bounds__(kT) sign_rows_kernel(const double* __restrict__ field, Rows g, IsoArg iso_arg,
                                                       uint32_t* __restrict__ bits, uint32_t* __restrict__ bad) {
    const double iso = iso_arg.get();
    const uint32_t lane = threadIdx.x & 31, row = blockIdx.x * (kT / 32) + (threadIdx.x >> 5);
    if (row >= g.n * g.n) return;
    const double* __restrict__ f = field + (uint64_t)row * g.n;
    bool broken = false;
#pragma unroll 4
    for (uint32_t w = 0; w < g.sign_words; ++w) {
        const uint32_t x = 32 * w + lane;
        const double v = x < g.n ? f[x] : 0.0;
        broken |= !isfinite(v);
        const uint32_t m = __ballot_sync(0xffffffffu, x < g.n && v < iso);
        if (lane == 0) bits[(uint64_t)row * g.sign_words + w] = m;
    }
    if (bad && broken) atomicOr(bad, 1u);
}

// *bad |= flag if a value is not finite.
__global__ void __launch_bounds__(kT) finite_kernel(const double* __restrict__ values, uint64_t count,
                                                    uint32_t* __restrict__ bad, uint32_t flag) {
    bool broken = false;
    const uint64_t stride = (uint64_t)gridDim.x * kT;
#pragma unroll 4
    for (uint64_t i = (uint64_t)blockIdx.x * kT + threadIdx.x; i < count; i += stride) broken |= !isfinite(values[i]);
    if (broken) atomicOr(bad, flag);
}

// Word t of each segment: active cells (corners on both sides, capi.mojo:946-960) and
// sign-changing edges of the three sweeps (capi.mojo:1090-1128: x-edges with y, z >= 1,
// y-edges with x, z >= 1, z-edges with x, y >= 1; coordinates below c).  An interior edge
// that changes sign lies on four active cells, so it always yields a quad.
__global__ void __launch_bounds__(kT) item_words_kernel(const uint32_t* __restrict__ bits, Rows g,
                                                        uint32_t* __restrict__ items) {
    const uint32_t t = blockIdx.x * kT + threadIdx.x;
    if (t >= g.segment) return;
    uint32_t out[4] = {0, 0, 0, 0};
    const uint32_t row = g.by_words.div(t), w = t - row * g.words;
    if (row < g.c * g.c) {
        const uint32_t z = g.by_c.div(row), y = row - z * g.c;
        uint32_t any = 0, all = ~0u, here = 0, shifted = 0, up_y = 0, up_z = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t at = ((uint64_t)(z + (k >> 1)) * g.n + y + (k & 1)) * g.sign_words + w;
            const uint32_t b = bits[at], next = w + 1 < g.sign_words ? bits[at + 1] : 0u, s = __funnelshift_r(b, next, 1);
            any |= b | s;
            all &= b & s;
            if (k == 0) {
                here = b;
                shifted = s;
            } else if (k == 1) up_y = b;
            else if (k == 2) up_z = b;
        }
        const uint32_t left = g.c - 32 * w, inside = left >= 32 ? ~0u : (1u << left) - 1u;
        const uint32_t inner = w == 0 ? inside & ~1u : inside;  // x >= 1
        out[0] = any & ~all & inside;
        if (y && z) out[1] = (here ^ shifted) & inside;
        if (z) out[2] = (here ^ up_y) & inner;
        if (y) out[3] = (here ^ up_z) & inner;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) items[(uint64_t)k * g.segment + t] = out[k];
}

__global__ void __launch_bounds__(kScanThreads) popcount_tiles_kernel(const uint32_t* __restrict__ items,
                                                                      uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t warp_sums[32];
    const uint4* __restrict__ p =
        reinterpret_cast<const uint4*>(items + (uint64_t)blockIdx.x * kTileWords) + 2 * threadIdx.x;
    const uint4 a = p[0], b = p[1];
    uint32_t total;
    block_exclusive_scan<uint32_t>(__popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w) + __popc(b.x) + __popc(b.y) +
                                       __popc(b.z) + __popc(b.w),
                                   warp_sums, total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}
static_assert(kScanItems == 8, "two uint4 per thread");

// tile_sums scanned: entry `tiles` of a segment is the number of cells, the last the number of items.
__global__ void store_counts_kernel(const uint32_t* __restrict__ tile_sums, uint32_t tiles, const uint32_t* total,
                                    const uint32_t* bad, int64_t* __restrict__ counts) {
    counts[0] = tile_sums[tiles];
    counts[1] = 2 * (int64_t)(*total - tile_sums[tiles]);  // two triangles per quad
    if (bad) counts[2] = *bad;
}

// Every item's place (kind, row and x) into the first slot of its output, in order, and the
// words' first cell ids.
__device__ __forceinline__ uint64_t place_of(uint32_t kind, uint32_t row, uint32_t x) {
    return ((uint64_t)kind << 60) | ((uint64_t)row << 16) | x;
}

__global__ void __launch_bounds__(kScanThreads) place_kernel(const uint32_t* __restrict__ items, Rows g, uint32_t tiles,
                                                             const uint32_t* __restrict__ tile_sums,
                                                             uint32_t* __restrict__ first,
                                                             uint64_t* __restrict__ vertex_slots,
                                                             uint64_t* __restrict__ face_slots) {
    __shared__ uint32_t warp_sums[32];
    const uint32_t kind = blockIdx.x / tiles, t0 = (blockIdx.x - kind * tiles) * kTileWords + threadIdx.x * kScanItems;
    const uint4* __restrict__ p = reinterpret_cast<const uint4*>(items + (uint64_t)kind * g.segment + t0);
    const uint4 a = p[0], b = p[1];
    const uint32_t word[kScanItems] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t sum = 0, total;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) sum += __popc(word[k]);
    uint32_t id = tile_sums[blockIdx.x] + block_exclusive_scan<uint32_t>(sum, warp_sums, total);
    const uint32_t cells = tile_sums[tiles];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        const uint32_t t = t0 + k;
        if (kind == 0) first[t] = id;
        uint32_t m = word[k];
        const uint32_t row = g.by_words.div(t), x0 = 32 * (t - row * g.words);
        while (m) {
            const uint64_t place = place_of(kind, row, x0 + __ffs(m) - 1);
            m &= m - 1;
            if (kind == 0) {
                if (vertex_slots) vertex_slots[id] = place;
            } else if (face_slots) {
                face_slots[6 * (uint64_t)(id - cells)] = place;
            }
            ++id;
        }
    }
}

__global__ void __launch_bounds__(kT) vertices_kernel(const double* __restrict__ field,
                                                      const double* __restrict__ density, Rows g, IsoArg iso_arg,
                                                      const uint32_t* __restrict__ cells, double* __restrict__ vertices,
                                                      double* __restrict__ vertex_density) {
    const uint32_t count = *cells;
    for (uint32_t id = blockIdx.x * kT + threadIdx.x; id < count; id += gridDim.x * kT) {
        const uint64_t place = reinterpret_cast<const uint64_t*>(vertex_density)[id];
        const uint32_t x = (uint32_t)place & 0xffffu, row = (uint32_t)(place >> 16), z = g.by_c.div(row), y = row - z * g.c;
        cell_vertex(field, density, g.n, x, y, z, iso_arg.get(), (double)g.c, vertices + 3 * (int64_t)id,
                    vertex_density + id);
    }
}

// One thread per quad: its two triangles (capi.mojo:1040-1071).
__global__ void __launch_bounds__(kT) quads_kernel(const uint32_t* __restrict__ bits, Rows g,
                                                   const uint32_t* __restrict__ items,
                                                   const uint32_t* __restrict__ first,
                                                   const uint32_t* __restrict__ cells, const uint32_t* __restrict__ total,
                                                   int64_t* __restrict__ faces) {
    const uint32_t count = *total - *cells;
    for (uint32_t quad = blockIdx.x * kT + threadIdx.x; quad < count; quad += gridDim.x * kT) {
        int64_t* out = faces + 6 * (int64_t)quad;
        const uint64_t place = (uint64_t)out[0];
        const uint32_t kind = (uint32_t)(place >> 60), x = (uint32_t)place & 0xffffu, row = (uint32_t)(place >> 16);
        const uint32_t z = g.by_c.div(row), y = row - z * g.c;
        const bool reverse = (bits[((uint64_t)z * g.n + y) * g.sign_words + (x >> 5)] >> (x & 31)) & 1u;
        auto cell = [&](uint32_t cx, uint32_t cy, uint32_t cz) -> int64_t {
            const uint32_t t = (cz * g.c + cy) * g.words + (cx >> 5);
            return (int64_t)first[t] + lanes_below(items[t], cx & 31);
        };
        int64_t a, b, c, d;
        if (kind == 1) {
            a = cell(x, y - 1, z - 1);
            b = cell(x, y, z - 1);
            c = cell(x, y, z);
            d = cell(x, y - 1, z);
        } else if (kind == 2) {
            a = cell(x - 1, y, z - 1);
            b = cell(x - 1, y, z);
            c = cell(x, y, z);
            d = cell(x, y, z - 1);
        } else {
            a = cell(x - 1, y - 1, z);
            b = cell(x, y - 1, z);
            c = cell(x, y, z);
            d = cell(x - 1, y, z);
        }
        out[0] = a;
        out[1] = reverse ? d : b;
        out[2] = c;
        out[3] = a;
        out[4] = c;
        out[5] = reverse ? b : d;
    }
}

// Arrays carved from the workspace, identically in count and emit.
struct Layout {
    Rows g;
    uint32_t tiles;  // scan tiles per segment
    uint32_t *bits, *items, *first, *tile_sums, *total, *bad;
    explicit Layout(int64_t n) : g(n), tiles(g.segment / kTileWords) {}
    void carve(Workspace& w) {
        bits = w.take<uint32_t>((size_t)g.n * g.n * g.sign_words);
        items = w.take<uint32_t>((size_t)4 * g.segment);
        first = w.take<uint32_t>(g.segment);
        tile_sums = w.take<uint32_t>((size_t)4 * tiles + 1);
        total = w.take<uint32_t>(1);
        bad = w.take<uint32_t>(1);
    }
};

inline size_t workspace_bytes(int64_t n) {
    if (n > kMaxSide) n = kMaxSide;
    return measure([&](Workspace& w) {
        Layout L(n);
        L.carve(w);
        scan_carve<uint32_t>(w, 4 * (int64_t)L.tiles);
    });
}

static int count_items(const double* field, const double* density, int64_t n, const double* iso, int64_t* counts,
                       bool checked, void* workspace, size_t bytes, cudaStream_t s) {
    if (n < 2 || n > kMaxSide || !field || !iso || !counts) return fail(PB_ERR_INVALID, "extract count: bad args");
    if (!workspace || bytes < workspace_bytes(n))
        return fail(PB_ERR_WORKSPACE, "extract: workspace needs %zu bytes", workspace_bytes(n));
    Workspace w(workspace, bytes);
    Layout L(n);
    L.carve(w);
    const Rows& g = L.g;
    if (checked) PB_CHECK_CUDA(cudaMemsetAsync(L.bad, 0, sizeof(uint32_t), s), "extract flags");
    sign_rows_kernel<<<(g.n * g.n + kT / 32 - 1) / (kT / 32), kT, 0, s>>>(field, g, IsoArg{0.0, iso}, L.bits,
                                                                          checked ? L.bad : nullptr);
    PB_CHECK_LAUNCH("sign_rows_kernel");
    if (checked && density) {
        const uint64_t nodes = (uint64_t)n * n * n;
        finite_kernel<<<(unsigned)std::min<uint64_t>((nodes + kT - 1) / kT, (uint64_t)kSMs * 16), kT, 0, s>>>(
            density, nodes, L.bad, 2u);
        PB_CHECK_LAUNCH("finite_kernel");
    }
    item_words_kernel<<<g.segment / kT, kT, 0, s>>>(L.bits, g, L.items);
    PB_CHECK_LAUNCH("item_words_kernel");
    popcount_tiles_kernel<<<4 * L.tiles, kScanThreads, 0, s>>>(L.items, L.tile_sums);
    PB_CHECK_LAUNCH("popcount_tiles_kernel");
    PB_TRY(exclusive_scan<uint32_t>(L.tile_sums, L.tile_sums, 4 * (int64_t)L.tiles, L.total, w, s));
    store_counts_kernel<<<1, 1, 0, s>>>(L.tile_sums, L.tiles, L.total, checked ? L.bad : nullptr, counts);
    PB_CHECK_LAUNCH("store_counts_kernel");
    return PB_OK;
}

}  // namespace fast

}  // namespace pb

using namespace pb;

extern "C" size_t pb_dual_workspace_size(int64_t n) { return dual_ws_bytes(n < 2 ? 2 : n); }

extern "C" int pb_dual_vertices_f64(const double* field, const double* density, int64_t n, double iso,
                                    int64_t* cell_map, double* vertices, double* vertex_density, int64_t capacity,
                                    int64_t* count, void* workspace, size_t workspace_bytes, void* stream) {
    return dual_vertices(field, density, n, IsoArg{iso, nullptr}, cell_map, vertices, vertex_density, capacity, count,
                         workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int pb_dual_vertices_f64_isoptr(const double* field, const double* density, int64_t n, const double* iso,
                                           int64_t* cell_map, double* vertices, double* vertex_density,
                                           int64_t capacity, int64_t* count, void* workspace, size_t workspace_bytes,
                                           void* stream) {
    if (!iso) return fail(PB_ERR_INVALID, "dual vertices: null iso pointer");
    return dual_vertices(field, density, n, IsoArg{0.0, iso}, cell_map, vertices, vertex_density, capacity, count,
                         workspace, workspace_bytes, (cudaStream_t)stream);
}

extern "C" int pb_dual_faces_f64(const double* field, int64_t n, double iso, const int64_t* cell_map, int64_t* faces,
                                 int64_t capacity, int64_t* count, void* workspace, size_t workspace_bytes,
                                 void* stream) {
    return dual_faces(field, n, IsoArg{iso, nullptr}, cell_map, faces, capacity, count, workspace, workspace_bytes,
                      (cudaStream_t)stream);
}

extern "C" int pb_dual_faces_f64_isoptr(const double* field, int64_t n, const double* iso, const int64_t* cell_map,
                                        int64_t* faces, int64_t capacity, int64_t* count, void* workspace,
                                        size_t workspace_bytes, void* stream) {
    if (!iso) return fail(PB_ERR_INVALID, "dual faces: null iso pointer");
    return dual_faces(field, n, IsoArg{0.0, iso}, cell_map, faces, capacity, count, workspace, workspace_bytes,
                      (cudaStream_t)stream);
}

// ---- extraction for reconstruct() (no counterpart in the reference's C API) ----
extern "C" size_t pb_extract_workspace_size(int64_t n) { return fast::workspace_bytes(n < 2 ? 2 : n); }

// Counts of the mesh extract_isosurface(field, iso) would give (capi.mojo:
// 798-1129): counts[0] = vertices, counts[1] = triangles (device int64[2]).
// Leaves in the workspace the state pb_extract_emit_f64 needs: call emit next
// with the same field, side, iso and workspace.  Sides 2..1025.
extern "C" int pb_extract_count_f64(const double* field, int64_t n, const double* iso, int64_t* counts,
                                    void* workspace, size_t workspace_bytes, void* stream) {
    return fast::count_items(field, nullptr, n, iso, counts, false, workspace, workspace_bytes, (cudaStream_t)stream);
}

// The same, and counts[2] (device int64[3]): 1 if a field value is not finite, plus 2 if a
// density value (density may be null) is not.
extern "C" int pb_extract_count_checked_f64(const double* field, const double* density, int64_t n, const double* iso,
                                            int64_t* counts, void* workspace, size_t workspace_bytes, void* stream) {
    return fast::count_items(field, density, n, iso, counts, true, workspace, workspace_bytes, (cudaStream_t)stream);
}

// Emits the counted mesh: vertices (counts[0] x 3), vertex_density
// (counts[0]), faces (counts[1] x 3), in the reference's order, bit-identical
// to pb_dual_vertices_f64 / pb_dual_faces_f64.  vertices (with
// vertex_density) or faces may be NULL when their count is 0; they are then
// not written.
extern "C" int pb_extract_emit_f64(const double* field, const double* density, int64_t n, const double* iso,
                                   double* vertices, double* vertex_density, int64_t* faces, void* workspace,
                                   size_t workspace_bytes, void* stream) {
    using namespace fast;
    if (n < 2 || n > kMaxSide || !field || !iso || (vertices && (!density || !vertex_density)))
        return fail(PB_ERR_INVALID, "extract emit: bad args");
    if (!workspace || workspace_bytes < fast::workspace_bytes(n))
        return fail(PB_ERR_WORKSPACE, "extract: workspace needs %zu bytes", fast::workspace_bytes(n));
    if (!vertices && !faces) return PB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    Workspace w(workspace, workspace_bytes);
    Layout L(n);
    L.carve(w);
    static_assert(sizeof(double) == sizeof(uint64_t) && sizeof(int64_t) == sizeof(uint64_t), "a place fits a slot");
    place_kernel<<<4 * L.tiles, kScanThreads, 0, s>>>(L.items, L.g, L.tiles, L.tile_sums, L.first,
                                                      vertices ? (uint64_t*)vertex_density : nullptr, (uint64_t*)faces);
    PB_CHECK_LAUNCH("place_kernel");
    const unsigned blocks = 16 * kSMs;  // grid-stride: the counts stay on the device
    if (vertices) {
        vertices_kernel<<<blocks, kT, 0, s>>>(field, density, L.g, IsoArg{0.0, iso}, L.tile_sums + L.tiles, vertices,
                                              vertex_density);
        PB_CHECK_LAUNCH("vertices_kernel");
    }
    if (faces) {
        quads_kernel<<<blocks, kT, 0, s>>>(L.bits, L.g, L.items, L.first, L.tile_sums + L.tiles, L.total, faces);
        PB_CHECK_LAUNCH("quads_kernel");
    }
    return PB_OK;
}
