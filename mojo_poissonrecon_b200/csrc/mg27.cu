// Galerkin coarse levels of the FP32 preconditioner.
//
// The reference's coarse levels rediscretise the operator (screen restricted
// and scaled by 4 per level, python/mojo_poissonrecon/core.py:267-269) and
// transfer with trilinear prolongation and boundary-normalised full weighting
// (src/capi.mojo:557-742).  The screening term pw*screen is concentrated on a
// thin shell of nodes around the samples, where it outweighs the Laplacian by
// one to two orders of magnitude; across that shell a trilinear coarse
// correction is wrong by O(1), and the reference-shaped cycle reduces the
// residual by only about 0.35 per cycle even with an exact coarse solve.  The
// FP32 preconditioner keeps the reference's fine operator and red-black
// smoother on level 0 and replaces the coarse side:
//   prolongation  P_s = S P, P trilinear, S = diag(s) with s_i = 1 where the
//                 fine node coincides with a coarse node, else
//                 s_i = (sum_{j != i} -a_ij) / a_ii  (deg / (deg + pw*screen)
//                 on level 0): a correction is damped where screening
//                 dominates the row;
//   restriction   R = P_s^T / 8 (full weighting scaled by s, not renormalised);
//   coarse ops    A_c = R A P_s (Galerkin), 27-point and symmetric;
//   coarsest      the 3^3 level solved exactly with its inverse.
// That cycle reduces the residual by about 0.03-0.05 per cycle independent of
// depth.  The FP64 outer loop still measures convergence with the reference's
// operator, so the answer is the reference's to the requested tolerance.
//
// Smoothing on 27-point levels: red-black ordered, same-colour couplings
// taken from the previous iterate (two passes per sweep, e_prev -> e_next,
// no in-place race); levels of side > 9 with their couplings packed per colour
// (see "packed 27-point levels" below), the smaller ones in one block.
//
// Storage of a 27-point level: 14 coefficient planes in the padded layout
// (level32.cuh), plane stride = padded_size(n); plane 0 the diagonal, planes
// 1..13 the couplings to the 13 "forward" neighbours J+K (K.z > 0; or K.z == 0
// and K.y > 0; or K = (1,0,0)).  The coupling to a backward neighbour J-K is
// plane k(K) at J-K (symmetry).  Ghost entries are zero.
#include <cuda_fp16.h>

#include "batch.cuh"
#include "common.cuh"
#include "level32.cuh"
#include "occupancy.cuh"

namespace pb {

__host__ __device__ constexpr bool is_forward(int dx, int dy, int dz) {
    return dz > 0 || (dz == 0 && (dy > 0 || (dy == 0 && dx > 0)));
}
__host__ __device__ constexpr int fwd_index(int dx, int dy, int dz) {
    return dz == 1 ? 1 + (dy + 1) * 3 + (dx + 1) : (dy == 1 ? 10 + (dx + 1) : 13);
}
__host__ __device__ constexpr float wt(int d) { return d == 0 ? 1.0f : 0.5f; }

__device__ __forceinline__ int64_t offset_of(const Geom& g, int dx, int dy, int dz) {
    return (int64_t)dx + (int64_t)dy * g.P + (int64_t)dz * g.plane;
}

// a(J, J+K) for the node at padded index p.
__device__ __forceinline__ float coupling(const float* __restrict__ c, int64_t cs, const Geom& g, int64_t p, int dx,
                                          int dy, int dz) {
    if (dx == 0 && dy == 0 && dz == 0) return c[p];
    if (is_forward(dx, dy, dz)) return c[fwd_index(dx, dy, dz) * cs + p];
    return c[fwd_index(-dx, -dy, -dz) * cs + p + offset_of(g, dx, dy, dz)];
}

__device__ __forceinline__ bool inside(int x, int y, int z, int n) {
    return (unsigned)x < (unsigned)n && (unsigned)y < (unsigned)n && (unsigned)z < (unsigned)n;
}

// Node of this thread on a level of side m, threads flattened over each plane's
// (x, y) (blockIdx.x) with the plane in blockIdx.y: full warps on 2^k + 1 sides.
// False past the plane's last node.
__device__ __forceinline__ bool plane_node(int m, int& x, int& y, int& z) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (unsigned)(m * m)) return false;
    y = (int)(t / (unsigned)m);
    x = (int)(t - (unsigned)y * m);
    z = blockIdx.y;
    return true;
}

inline dim3 plane_grid(int m, int threads) { return dim3((m * m + threads - 1) / threads, m); }

// ---- Galerkin product A_c = P_s^T A P_s / 8 from level 0 ------------------------
// One thread per coarse node J streams once over the fine nodes i = 2J + o of
// J's support (27) and their 7-point stencil neighbours j = i + K, and
// scatters the product p_iJ a_ij s_j into the stored entries A_c[J, J+m]
// (m = 0 or forward) whose column support holds j, with weight P(d - 2m),
// d = o + K.  Every index and weight is resolved at compile time, so the 14
// sums stay in registers.  (From a 27-point level the product is separable:
// see the x, y, z stages below.)
__device__ __forceinline__ void scatter14(float v, int dx, int dy, int dz, float* acc) {
#pragma unroll
    for (int mz = -1; mz <= 1; ++mz)
#pragma unroll
        for (int my = -1; my <= 1; ++my)
#pragma unroll
            for (int mx = -1; mx <= 1; ++mx) {
                const int ex = dx - 2 * mx, ey = dy - 2 * my, ez = dz - 2 * mz;
                if (ex < -1 || ex > 1 || ey < -1 || ey > 1 || ez < -1 || ez > 1) continue;
                const bool centre = mx == 0 && my == 0 && mz == 0;
                if (!centre && !is_forward(mx, my, mz)) continue;
                acc[centre ? 0 : fwd_index(mx, my, mz)] += v * (wt(ex) * wt(ey) * wt(ez));
            }
}

// The sums for one coarse node below level 0: `D` is the level-0 diagonal
// (couplings -h2 to in-grid face neighbours), S its prolongation weights.
// INTERIOR: every i and j of J lies in the grid (no bounds tests).
template <bool INTERIOR>
__device__ __forceinline__ void galerkin7_sums(const float* __restrict__ D, const float* __restrict__ S,
                                               const Geom& gf, float h2, int xc, int yc, int zc, float* acc) {
    const int fn = gf.n;
#pragma unroll
    for (int oz = -1; oz <= 1; ++oz)
#pragma unroll
        for (int oy = -1; oy <= 1; ++oy)
#pragma unroll
            for (int ox = -1; ox <= 1; ++ox) {
                const int xi = 2 * xc + ox, yi = 2 * yc + oy, zi = 2 * zc + oz;
                if (!INTERIOR && !inside(xi, yi, zi, fn)) continue;
                const int64_t pi = gf.at(xi, yi, zi);
                const float si = wt(ox) * wt(oy) * wt(oz) * S[pi];
#pragma unroll
                for (int kz = -1; kz <= 1; ++kz)
#pragma unroll
                    for (int ky = -1; ky <= 1; ++ky)
#pragma unroll
                        for (int kx = -1; kx <= 1; ++kx) {
                            if ((kx != 0) + (ky != 0) + (kz != 0) > 1) continue;  // 7-point stencil
                            if (!INTERIOR && !inside(xi + kx, yi + ky, zi + kz, fn)) continue;
                            const float a = (kx == 0 && ky == 0 && kz == 0) ? D[pi] : -h2;
                            scatter14(si * a * S[pi + offset_of(gf, kx, ky, kz)], ox + kx, oy + ky, oz + kz, acc);
                        }
            }
}

__device__ __forceinline__ void galerkin_store(const float* acc, float* __restrict__ cc, int64_t cs, const Geom& gc,
                                               int xc, int yc, int zc) {
    const int64_t p = gc.at(xc, yc, zc);
    cc[p] = acc[0] * 0.125f;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx)
                if (is_forward(dx, dy, dz)) {
                    const int k = fwd_index(dx, dy, dz);
                    cc[k * cs + p] = inside(xc + dx, yc + dy, zc + dz, gc.n) ? acc[k] * 0.125f : 0.0f;
                }
}

// The interior sums where the weights are 1 and the diagonal is 6 h^-2: multiples of a
// power of two, exact in any order.
struct Plain14 {
    float sum[14];
    explicit Plain14(float h2) {
        for (float& v : sum) v = 0.0f;
        for (int o = 0; o < 27; ++o) {
            const int ox = o % 3 - 1, oy = o / 3 % 3 - 1, oz = o / 9 - 1;
            for (int k = 0; k < 27; ++k) {
                const int kx = k % 3 - 1, ky = k / 3 % 3 - 1, kz = k / 9 - 1;
                if ((kx != 0) + (ky != 0) + (kz != 0) > 1) continue;
                const float v = wt(ox) * wt(oy) * wt(oz) * (k == 13 ? 6.0f * h2 : -h2);
                for (int m = 13; m < 27; ++m) {  // the centre and what lies forward of it
                    const int mx = m % 3 - 1, my = m / 3 % 3 - 1, mz = m / 9 - 1;
                    const int ex = ox + kx - 2 * mx, ey = oy + ky - 2 * my, ez = oz + kz - 2 * mz;
                    if (ex * ex <= 1 && ey * ey <= 1 && ez * ez <= 1)
                        sum[m == 13 ? 0 : fwd_index(mx, my, mz)] += v * (wt(ex) * wt(ey) * wt(ez));
                }
            }
        }
    }
};

// Level 0 as the fine level: interior coarse nodes take the branch-free sums, and those
// without screening among the 5^3 fine nodes around them (most: it lies around the
// samples) the same constants: bound by the 14 stores there instead of by the 189 loads
// and 1,500 operations of the sums.  257^3, 1M points: 210 -> 144 us (a warp
// of 32 coarse x runs the sums if any of its nodes has to); 513^3, 2M: 1,440 -> 788.
__global__ void __launch_bounds__(128) galerkin7_kernel(const float* __restrict__ D, const float* __restrict__ S,
                                                        const uint32_t* __restrict__ screened, const Plain14 plain,
                                                        Geom gf, float h2, float* __restrict__ cc, int64_t cs,
                                                        Geom gc) {
    const int cn = gc.n;
    int xc, yc, zc;
    if (!plane_node(cn, xc, yc, zc)) return;
    float acc[14];
    const bool interior = xc >= 1 && yc >= 1 && zc >= 1 && xc <= cn - 2 && yc <= cn - 2 && zc <= cn - 2;
    if (interior && five_cubed_empty(screened, gf.n, 2 * xc, 2 * yc, 2 * zc)) {
#pragma unroll
        for (int k = 0; k < 14; ++k) acc[k] = plain.sum[k];
    } else {
#pragma unroll
        for (int k = 0; k < 14; ++k) acc[k] = 0.0f;
        if (interior) galerkin7_sums<true>(D, S, gf, h2, xc, yc, zc, acc);
        else galerkin7_sums<false>(D, S, gf, h2, xc, yc, zc, acc);
    }
    galerkin_store(acc, cc, cs, gc, xc, yc, zc);
}

// ---- separable product for a 27-point fine level ---------------------------------
// P is the tensor product of 1D linear interpolation (coarse M -> fine j with
// weight 1 at j = 2M and 1/2 at j = 2M +- 1), so P^T (S A S) P / 8 contracts
// one axis at a time: x, then y, then z.  Each stage maps fine positions 2M +
// a (a in {-1, 0, 1}) and their offsets d to coarse offsets m with weights
// P(a) P(a + d - 2m), keeping the other two axes' offsets, and takes 81
// products per output node against the direct sum's 27 x 27 per coarse node
// scattered over 14 entries.  Stages x and y write full 27-entry stencils,
// entry e = (oz+1)*9 + (oy+1)*3 + (ox+1), as 27 planes of a dense grid into
// scratch, a slab of fine z-planes at a time; stage z writes the 14 stored
// planes.  Out-of-grid fine nodes and neighbours contribute nothing.
__host__ __device__ constexpr float wt1(int d) { return d == 0 ? 1.0f : (d == 1 || d == -1 ? 0.5f : 0.0f); }

// Stage x: node (I, y, z) of the grid cn x fn x (slab of fine z from zlo);
// entry (m, dy, dz) = sum over a, dx of P(a) s_i a(i, j) s_j P(a + dx - 2m),
// i = (2I + a, y, z), j = i + (dx, dy, dz).
__global__ void __launch_bounds__(128) galerkin_x_kernel(const float* __restrict__ c, int64_t cs,
                                                         const float* __restrict__ S, Geom gf, int cn, int zlo,
                                                         float* __restrict__ out, int64_t ps) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;  // flattened over (I, y)
    const int fn = gf.n;
    if (t >= (unsigned)(cn * fn)) return;
    const int y = (int)(t / (unsigned)cn), I = (int)(t - (unsigned)y * cn);
    const int z = zlo + blockIdx.y;
    const int64_t o = ((int64_t)blockIdx.y * fn + y) * cn + I;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
            float acc[3] = {0.0f, 0.0f, 0.0f};
            if (inside(0, y + dy, z + dz, fn)) {
#pragma unroll
                for (int a = -1; a <= 1; ++a) {
                    const int xi = 2 * I + a;
                    if (xi < 0 || xi >= fn) continue;
                    const int64_t pi = gf.at(xi, y, z);
                    const float si = wt1(a) * S[pi];
#pragma unroll
                    for (int dx = -1; dx <= 1; ++dx) {
                        if (xi + dx < 0 || xi + dx >= fn) continue;
                        const float t = si * coupling(c, cs, gf, pi, dx, dy, dz) * S[pi + offset_of(gf, dx, dy, dz)];
#pragma unroll
                        for (int m = -1; m <= 1; ++m)
                            if (wt1(a + dx - 2 * m) != 0.0f) acc[m + 1] += t * wt1(a + dx - 2 * m);
                    }
                }
            }
#pragma unroll
            for (int m = -1; m <= 1; ++m) out[((dz + 1) * 9 + (dy + 1) * 3 + (m + 1)) * ps + o] = acc[m + 1];
        }
}

// Stage y: node (I, J, z) of cn x cn x slab from stage x's cn x fn x slab.
__global__ void __launch_bounds__(128) galerkin_y_kernel(const float* __restrict__ in, int64_t pin, int fn, int cn,
                                                         float* __restrict__ out, int64_t pout) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;  // flattened over (I, J)
    if (t >= (unsigned)(cn * cn)) return;
    const int J = (int)(t / (unsigned)cn), I = (int)(t - (unsigned)J * cn);
    const int zr = blockIdx.y;
    const int64_t o = ((int64_t)zr * cn + J) * cn + I;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int m = -1; m <= 1; ++m) {
            float acc[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int b = -1; b <= 1; ++b) {
                const int yj = 2 * J + b;
                if (yj < 0 || yj >= fn) continue;
                const int64_t q = ((int64_t)zr * fn + yj) * cn + I;
#pragma unroll
                for (int dy = -1; dy <= 1; ++dy) {
                    const float v = wt1(b) * in[((dz + 1) * 9 + (dy + 1) * 3 + (m + 1)) * pin + q];
#pragma unroll
                    for (int my = -1; my <= 1; ++my)
                        if (wt1(b + dy - 2 * my) != 0.0f) acc[my + 1] += v * wt1(b + dy - 2 * my);
                }
            }
#pragma unroll
            for (int my = -1; my <= 1; ++my) out[((dz + 1) * 9 + (my + 1) * 3 + (m + 1)) * pout + o] = acc[my + 1];
        }
}

// Stage z: coarse node (I, J, K), K in [k0, k1), from stage y's slab (fine z
// from zlo, nz planes); the diagonal and the 13 forward couplings / 8 into the
// 14 planes, zero where the coarse neighbour lies outside the grid.
__global__ void __launch_bounds__(128) galerkin_z_kernel(const float* __restrict__ in, int64_t pin, int fn, int zlo,
                                                         int k0, float* __restrict__ cc, int64_t cs, Geom gc) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;  // flattened over (I, J)
    const int cn = gc.n;
    if (t >= (unsigned)(cn * cn)) return;
    const int J = (int)(t / (unsigned)cn), I = (int)(t - (unsigned)J * cn);
    const int K = k0 + blockIdx.y;
    const int64_t p = gc.at(I, J, K);
#pragma unroll
    for (int my = -1; my <= 1; ++my)
#pragma unroll
        for (int m = -1; m <= 1; ++m) {
            float acc[3] = {0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = -1; c <= 1; ++c) {
                const int zf = 2 * K + c;
                if (zf < 0 || zf >= fn) continue;
                const int64_t q = ((int64_t)(zf - zlo) * cn + J) * cn + I;
#pragma unroll
                for (int dz = -1; dz <= 1; ++dz) {
                    const float v = wt1(c) * in[((dz + 1) * 9 + (my + 1) * 3 + (m + 1)) * pin + q];
#pragma unroll
                    for (int mz = -1; mz <= 1; ++mz)
                        if (wt1(c + dz - 2 * mz) != 0.0f) acc[mz + 1] += v * wt1(c + dz - 2 * mz);
                }
            }
#pragma unroll
            for (int mz = -1; mz <= 1; ++mz) {
                const bool centre = m == 0 && my == 0 && mz == 0;
                if (!centre && !is_forward(m, my, mz)) continue;
                const float val = inside(I + m, J + my, K + mz, cn) ? acc[mz + 1] * 0.125f : 0.0f;
                cc[(centre ? 0 : fwd_index(m, my, mz)) * cs + p] = val;
            }
        }
}

// The same product for a small coarse level, one warp per coarse node: a lane takes one
// fine node i of the support, contracts its 27 couplings axis by axis with the weights
// P(o + d - 2m) of its own place, and the lanes' sums are added.  Below some size the
// three stages take 6 to 8 us each however small the level; this takes 12 us at coarse
// side 17 and 5 below it, but 55 at 33 against 37 for the stages.
constexpr int kSmallCoarse = 17;

__global__ void __launch_bounds__(128) galerkin_small_kernel(const float* __restrict__ c, int64_t cs,
                                                             const float* __restrict__ S, Geom gf,
                                                             float* __restrict__ cc, int64_t ccs, Geom gc) {
    const int cn = gc.n, lane = threadIdx.x & 31;
    const int node = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (node >= cn * cn * cn) return;  // whole warps
    const int I = node % cn, J = node / cn % cn, K = node / (cn * cn);
    const int o[3] = {lane % 3 - 1, lane / 3 % 3 - 1, lane / 9 - 1};
    const int xi = 2 * I + o[0], yi = 2 * J + o[1], zi = 2 * K + o[2];
    float sum[14] = {};
    if (lane < 27 && inside(xi, yi, zi, gf.n)) {  // couplings and weights outside the grid are zero
        float w[3][3][3];  // per axis: P(o + d - 2m) by d, m
#pragma unroll
        for (int axis = 0; axis < 3; ++axis)
#pragma unroll
            for (int d = 0; d < 3; ++d)
#pragma unroll
                for (int m = 0; m < 3; ++m) w[axis][d][m] = wt1(o[axis] + (d - 1) - 2 * (m - 1));
        const int64_t p = gf.at(xi, yi, zi);
        const float si = wt1(o[0]) * wt1(o[1]) * wt1(o[2]) * S[p];
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
            float xy[3][3] = {};  // by my, mx
#pragma unroll
            for (int dy = 0; dy < 3; ++dy) {
                float x[3] = {};
#pragma unroll
                for (int dx = 0; dx < 3; ++dx) {
                    const float t = si * coupling(c, cs, gf, p, dx - 1, dy - 1, dz - 1) *
                                    S[p + offset_of(gf, dx - 1, dy - 1, dz - 1)];
#pragma unroll
                    for (int m = 0; m < 3; ++m) x[m] += t * w[0][dx][m];
                }
#pragma unroll
                for (int my = 0; my < 3; ++my)
#pragma unroll
                    for (int mx = 0; mx < 3; ++mx) xy[my][mx] += x[mx] * w[1][dy][my];
            }
#pragma unroll
            for (int mz = 1; mz < 3; ++mz)
#pragma unroll
                for (int my = 0; my < 3; ++my)
#pragma unroll
                    for (int mx = 0; mx < 3; ++mx) {
                        const bool centre = mx == 1 && my == 1 && mz == 1;
                        if (centre || is_forward(mx - 1, my - 1, mz - 1))
                            sum[centre ? 0 : fwd_index(mx - 1, my - 1, mz - 1)] += xy[my][mx] * w[2][dz][mz];
                    }
        }
    }
    const int64_t q = gc.at(I, J, K);
#pragma unroll
    for (int k = 0; k < 14; ++k) {
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], step);
    }
    if (lane == 0) cc[q] = sum[0] * 0.125f;
#pragma unroll
    for (int m = 14; m < 27; ++m) {  // forward neighbours, a lane each
        const int mx = m % 3 - 1, my = m / 3 % 3 - 1, mz = m / 9 - 1, k = fwd_index(mx, my, mz);
        if (lane == k) cc[k * ccs + q] = inside(I + mx, J + my, K + mz, cn) ? sum[k] * 0.125f : 0.0f;
    }
}

// A 7-point level (diagonal D, off-diagonals -h2 inside the grid) as 14 planes.
__global__ void level7_to_27_kernel(const float* __restrict__ D, Geom g, float h2, float* __restrict__ c, int64_t cs) {
    const int n = g.n;
    int x, y, z;
    if (!plane_node(n, x, y, z)) return;
    const int64_t p = g.at(x, y, z);
    c[p] = D[p];
#pragma unroll
    for (int k = 1; k <= 13; ++k) c[k * cs + p] = 0.0f;
    c[fwd_index(1, 0, 0) * cs + p] = x + 1 < n ? -h2 : 0.0f;
    c[fwd_index(0, 1, 0) * cs + p] = y + 1 < n ? -h2 : 0.0f;
    c[fwd_index(0, 0, 1) * cs + p] = z + 1 < n ? -h2 : 0.0f;
}

// 1/a_JJ and the prolongation weight s_J of a 27-point level.
__global__ void level27_finish_kernel(const float* __restrict__ c, int64_t cs, Geom g, float* __restrict__ invD,
                                      float* __restrict__ fac) {
    const int n = g.n;
    int x, y, z;
    if (!plane_node(n, x, y, z)) return;
    const int64_t p = g.at(x, y, z);
    float off = 0.0f;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx)
                if (dx || dy || dz) off -= coupling(c, cs, g, p, dx, dy, dz);
    const float d = c[p];
    invD[p] = 1.0f / d;
    float s = 1.0f;
    if ((x | y | z) & 1) s = fminf(fmaxf(off / d, 0.0f), 1.0f);
    fac[p] = s;
}

// ---- 27-point smoothing, residual, transfers ------------------------------------
// coarse[J] = sum_o w(o)/64 res[2J+o], w = prod (2 on the axis, 1 off it);
// out-of-grid fine nodes are ghosts holding zero.
__device__ __forceinline__ void restrict27_body(const float* __restrict__ res, Geom gf, float* __restrict__ coarse,
                                                Geom gc, int bx, int by) {
    const unsigned t = bx * blockDim.x + threadIdx.x;
    if (t >= (unsigned)(gc.n * gc.n)) return;
    const int y = (int)(t / (unsigned)gc.n), x = (int)(t - (unsigned)y * gc.n), z = by;
    const int64_t p = gf.at(2 * x, 2 * y, 2 * z);
    float s = 0.0f;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx)
                s += res[p + offset_of(gf, dx, dy, dz)] * (float)((dx ? 1 : 2) * (dy ? 1 : 2) * (dz ? 1 : 2));
    coarse[gc.at(x, y, z)] = s * (1.0f / 64.0f);
}

__global__ void __launch_bounds__(256) restrict27_kernel(const float* __restrict__ res, Geom gf,
                                                         float* __restrict__ coarse, Geom gc) {
    restrict27_body(res, gf, coarse, gc, blockIdx.x, blockIdx.y);
}

// ---- packed 27-point levels: per-colour FP16 couplings --------------------------
// A colour pass over the 14-plane storage reads its nodes' forward coupling
// planes with stride 2 and the backward couplings at neighbours: about 140
// bytes per node and sweep from DRAM on the 129^3 level.  Packed, each colour's nodes are
// numbered compactly (row (y, z), i-th node of the colour: x = 2i + ((y+z+c)&1),
// compact index (z*n + y)*Pc + i, Pc = (n+1)/2) and hold their 26 couplings
// divided by the diagonal, c_K = -a(J, J+K) / a(J, J), in FP16 (|c_K| <= 1),
// node-major: 32 halves (64 bytes, the last 6 zero) per node, coupling k =
// offset index over (dz, dy, dx) in lexicographic order with the centre
// skipped, read as four 16-byte loads; and 1/a(J, J) in FP32.  Relaxation and residual of the level both
// use the rounded couplings, so the level's operator stays one operator:
//   e_new(J) = invD(J) rhs(J) + sum_K c_K e(J+K)
//   r(J)     = rhs(J) - (e(J) - sum_K c_K e(J+K)) / invD(J)
// The rounding (relative 2^-11) changes the preconditioner only; convergence is
// measured with the reference's FP64 operator.
__host__ __device__ constexpr int packed_index(int dx, int dy, int dz) {
    const int k = (dz + 1) * 9 + (dy + 1) * 3 + (dx + 1);
    return k < 13 ? k : k - 1;  // the centre (13) is not stored
}

constexpr int kPackedStride = 32;  // halves per node

struct Packed {
    int n, Pc;
    int64_t cs;  // compact nodes per colour = n * n * Pc
    __host__ __device__ __forceinline__ int64_t at(int i, int y, int z) const { return ((int64_t)z * n + y) * Pc + i; }
};

__host__ __device__ inline Packed packed_of(int n) {
    Packed p;
    p.n = n;
    p.Pc = (n + 1) / 2;
    p.cs = (int64_t)n * n * p.Pc;
    return p;
}

__global__ void __launch_bounds__(256) pack27_kernel(const float* __restrict__ c, int64_t cs, Geom g, Packed pk,
                                                     __half* __restrict__ h0, __half* __restrict__ h1,
                                                     float* __restrict__ i0, float* __restrict__ i1) {
    const int n = g.n;
    int x, y, z;
    if (!plane_node(n, x, y, z)) return;
    const int colour = (x + y + z) & 1;
    const int64_t q = pk.at(x >> 1, y, z);
    const int64_t p = g.at(x, y, z);
    const float inv = 1.0f / c[p];
    (colour ? i1 : i0)[q] = inv;
    __align__(16) __half v[kPackedStride];
#pragma unroll
    for (int k = 26; k < kPackedStride; ++k) v[k] = __float2half_rn(0.0f);
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (!(dx || dy || dz)) continue;
                v[packed_index(dx, dy, dz)] = __float2half_rn(-coupling(c, cs, g, p, dx, dy, dz) * inv);
            }
    uint4* dst = reinterpret_cast<uint4*>((colour ? h1 : h0) + q * kPackedStride);
    const uint4* src = reinterpret_cast<const uint4*>(v);
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[k] = src[k];
}

// The 26 couplings of compact node q, as floats.
__device__ __forceinline__ void load_couplings(const __half* __restrict__ h, int64_t q, float* c) {
    const uint4* src = reinterpret_cast<const uint4*>(h + q * kPackedStride);
    __align__(16) __half v[kPackedStride];
    uint4* d = reinterpret_cast<uint4*>(v);
#pragma unroll
    for (int k = 0; k < 4; ++k) d[k] = src[k];
#pragma unroll
    for (int k = 0; k < 26; ++k) c[k] = __half2float(v[k]);
}

// One colour pass on a packed level: nodes of colour COLOUR get
// invD rhs + sum_K c_K e(J+K), neighbours of the other colour read from `next`
// when COLOUR == 1 (updated by pass 0), everything else from `prev` (zero when
// ZERO).
template <int COLOUR, bool ZERO>
__device__ __forceinline__ void relax27p_body(const float* __restrict__ prev, float* next,
                                              const float* __restrict__ rhs, const __half* __restrict__ h,
                                              const float* __restrict__ inv, Geom g, Packed pk, int bx, int by) {
    // threads flattened over the plane's compact (i, y) nodes: full warps on odd rows
    const unsigned t = bx * blockDim.x + threadIdx.x;
    const int n = g.n, z = by;
    if (t >= (unsigned)(pk.Pc * n)) return;
    const int y = (int)(t / (unsigned)pk.Pc), i = (int)(t - (unsigned)y * pk.Pc);
    const int x = 2 * i + ((y + z + COLOUR) & 1);
    if (x >= n) return;
    const int64_t p = g.at(x, y, z), q = pk.at(i, y, z);
    float cf[26];
    load_couplings(h, q, cf);
    float s = 0.0f;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (!(dx || dy || dz)) continue;
                const bool other = ((dx + dy + dz) & 1) != 0;
                if (ZERO && !(COLOUR == 1 && other)) continue;
                const int64_t o = p + offset_of(g, dx, dy, dz);
                const float v = (COLOUR == 1 && other) ? next[o] : prev[o];
                s += cf[packed_index(dx, dy, dz)] * v;
            }
    next[p] = inv[q] * rhs[p] + s;
}

template <int COLOUR, bool ZERO>
__global__ void __launch_bounds__(256) relax27p_kernel(const float* __restrict__ prev, float* next,
                                                       const float* __restrict__ rhs, const __half* __restrict__ h,
                                                       const float* __restrict__ inv, Geom g, Packed pk) {
    relax27p_body<COLOUR, ZERO>(prev, next, rhs, h, inv, g, pk, blockIdx.x, blockIdx.y);
}

// The same colour pass with the neighbour planes staged in shared memory.  A
// block owns 32 compact columns (64 x) by 8 rows of the colour's nodes and
// marches `tz` planes; each plane of `prev` (and, for the colour-1 pass, the
// colour-0 values of `next`) over the tile and its one-node halo is loaded
// once, coalesced, into a ring of four planes, so a node reads its 26
// neighbours from shared memory instead of 26 gathers.  Out-of-grid halo
// entries read zero, as the ghosts do.  Same values, same summation order:
// results are bit-identical to relax27p_kernel.
constexpr int kTPi = 32, kTPy = 8, kTPRing = 4;
constexpr int kTPW = 2 * kTPi + 4, kTPH = kTPy + 2;  // staged x from 2 i0 - 2, y from y0 - 1

template <int COLOUR, bool ZERO>
__global__ void __launch_bounds__(kTPi* kTPy) relax27p_tiled_kernel(const float* __restrict__ prev, float* next,
                                                                    const float* __restrict__ rhs,
                                                                    const __half* __restrict__ h,
                                                                    const float* __restrict__ inv, Geom g, Packed pk,
                                                                    int tz) {
    constexpr bool kPrev = !ZERO, kNext = COLOUR == 1;
    __shared__ float sp[kPrev ? kTPRing : 1][kTPH][kTPW];
    __shared__ float sn[kNext ? kTPRing : 1][kTPH][kTPW];
    const int n = g.n;
    const int i0 = blockIdx.x * kTPi, y0 = blockIdx.y * kTPy;
    const int z0 = blockIdx.z * tz, z1 = min(n, z0 + tz);
    const int tid = threadIdx.x, ti = tid % kTPi, ty = tid / kTPi;
    const int xs0 = 2 * i0 - 2, ys0 = y0 - 1;
    auto stage = [&](int z) {  // plane z (>= -1) into ring slot (z + 1) % kTPRing
        const int slot = (z + 1) % kTPRing;
        for (int k = tid; k < kTPH * kTPW; k += kTPi * kTPy) {
            const int ry = k / kTPW, rx = k - ry * kTPW;
            const int x = xs0 + rx, y = ys0 + ry;
            const bool ok = x >= -1 && x <= n && y >= -1 && y <= n && z <= n;
            const int64_t o = ok ? g.at(x, y, z) : 0;
            if (kPrev) sp[kPrev ? slot : 0][ry][rx] = ok ? prev[o] : 0.0f;
            if (kNext) sn[kNext ? slot : 0][ry][rx] = ok && ((x + y + z) & 1) != COLOUR ? next[o] : 0.0f;
        }
    };
    if (kPrev || kNext) {
        stage(z0 - 1);
        stage(z0);
    }
    const int i = i0 + ti, y = y0 + ty;
    for (int z = z0; z < z1; ++z) {
        if (kPrev || kNext) {
            if (z + 1 <= n) stage(z + 1);  // into the slot of plane z - 3, last read before the previous barrier
            __syncthreads();
        }
        if (i >= pk.Pc || y >= n) continue;
        const int x = 2 * i + ((y + z + COLOUR) & 1);
        if (x >= n) continue;
        const int64_t p = g.at(x, y, z), q = pk.at(i, y, z);
        float cf[26];
        load_couplings(h, q, cf);
        float s = 0.0f;
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx) {
                    if (!(dx || dy || dz)) continue;
                    const bool other = ((dx + dy + dz) & 1) != 0;
                    if (ZERO && !(COLOUR == 1 && other)) continue;
                    const int sl = (z + dz + 1) % kTPRing, ry = ty + 1 + dy, rx = x + dx - xs0;
                    const float v = (COLOUR == 1 && other) ? sn[kNext ? sl : 0][ry][rx] : sp[kPrev ? sl : 0][ry][rx];
                    s += cf[packed_index(dx, dy, dz)] * v;
                }
        next[p] = inv[q] * rhs[p] + s;
    }
}

// res = s (rhs - A e) on a packed level, one thread per node.
__device__ __forceinline__ void residual27p_body(const float* __restrict__ e, const float* __restrict__ rhs,
                                                 const __half* __restrict__ h0, const __half* __restrict__ h1,
                                                 const float* __restrict__ i0, const float* __restrict__ i1,
                                                 const float* __restrict__ fac, Geom g, Packed pk,
                                                 float* __restrict__ res, int bx, int by) {
    const unsigned t = bx * blockDim.x + threadIdx.x;  // flattened over the plane's (x, y)
    const int n = g.n, z = by;
    if (t >= (unsigned)(n * n)) return;
    const int y = (int)(t / (unsigned)n), x = (int)(t - (unsigned)y * n);
    const int colour = (x + y + z) & 1;
    const __half* __restrict__ h = colour ? h1 : h0;
    const int64_t p = g.at(x, y, z), q = pk.at(x >> 1, y, z);
    float cf[26];
    load_couplings(h, q, cf);
    float s = 0.0f;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (!(dx || dy || dz)) continue;
                s += cf[packed_index(dx, dy, dz)] * e[p + offset_of(g, dx, dy, dz)];
            }
    const float inv = colour ? i1[q] : i0[q];
    res[p] = fac[p] * (rhs[p] - (e[p] - s) / inv);
}

__global__ void __launch_bounds__(256) residual27p_kernel(const float* __restrict__ e, const float* __restrict__ rhs,
                                                          const __half* __restrict__ h0,
                                                          const __half* __restrict__ h1,
                                                          const float* __restrict__ i0, const float* __restrict__ i1,
                                                          const float* __restrict__ fac, Geom g, Packed pk,
                                                          float* __restrict__ res) {
    residual27p_body(e, rhs, h0, h1, i0, i1, fac, g, pk, res, blockIdx.x, blockIdx.y);
}

// The packed residual with e's planes staged in shared memory: a block owns a
// 64 x 4 tile of nodes (both colours) and marches `tz` planes with a ring of
// four planes of e over the tile and its halo; same values and order as
// residual27p_kernel, so bit-identical results.
constexpr int kTRx = 64, kTRy = 4;
constexpr int kTRW = kTRx + 4, kTRH = kTRy + 2;  // staged x from x0 - 2, y from y0 - 1

__global__ void __launch_bounds__(kTRx* kTRy) residual27p_tiled_kernel(
    const float* __restrict__ e, const float* __restrict__ rhs, const __half* __restrict__ h0,
    const __half* __restrict__ h1, const float* __restrict__ i0, const float* __restrict__ i1,
    const float* __restrict__ fac, Geom g, Packed pk, float* __restrict__ res, int tz) {
    __shared__ float se[kTPRing][kTRH][kTRW];
    const int n = g.n;
    const int x0 = blockIdx.x * kTRx, y0 = blockIdx.y * kTRy;
    const int z0 = blockIdx.z * tz, z1 = min(n, z0 + tz);
    const int tid = threadIdx.x, tx = tid % kTRx, ty = tid / kTRx;
    const int xs0 = x0 - 2, ys0 = y0 - 1;
    auto stage = [&](int z) {
        const int slot = (z + 1) % kTPRing;
        for (int k = tid; k < kTRH * kTRW; k += kTRx * kTRy) {
            const int ry = k / kTRW, rx = k - ry * kTRW;
            const int x = xs0 + rx, y = ys0 + ry;
            const bool ok = x >= -1 && x <= n && y >= -1 && y <= n && z <= n;
            se[slot][ry][rx] = ok ? e[g.at(x, y, z)] : 0.0f;
        }
    };
    stage(z0 - 1);
    stage(z0);
    const int x = x0 + tx, y = y0 + ty;
    for (int z = z0; z < z1; ++z) {
        if (z + 1 <= n) stage(z + 1);
        __syncthreads();
        if (x >= n || y >= n) continue;
        const int colour = (x + y + z) & 1;
        const __half* __restrict__ h = colour ? h1 : h0;
        const int64_t p = g.at(x, y, z), q = pk.at(x >> 1, y, z);
        float cf[26];
        load_couplings(h, q, cf);
        float s = 0.0f;
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
            for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
                for (int dx = -1; dx <= 1; ++dx) {
                    if (!(dx || dy || dz)) continue;
                    s += cf[packed_index(dx, dy, dz)] * se[(z + dz + 1) % kTPRing][ty + 1 + dy][tx + 2 + dx];
                }
        const float inv = colour ? i1[q] : i0[q];
        res[p] = fac[p] * (rhs[p] - (se[(z + 1) % kTPRing][ty + 1][tx + 2] - s) / inv);
    }
}

// ---- exact solve on the 3^3 level -----------------------------------------------
// The 27 x 27 operator of the coarsest level inverted once per set-up by one
// block: FP64 Gauss-Jordan without pivoting (the Galerkin operator is
// symmetric positive definite), a thread per element, the pivot's row and column
// through shared memory (two by step parity: one barrier a step); stored FP64 row-major
// and applied in FP64 (the coarsest-level solve stays in double precision).  One warp
// with a row per lane took 27 us, mostly a serial walk of the rows.
constexpr int kInvN = 27;

__global__ void __launch_bounds__(32 * kInvN) coarse_inverse_kernel(const float* __restrict__ c, int64_t cs, Geom g,
                                                                    double* __restrict__ inv) {
    __shared__ double pivot_row[2][32], pivot_column[2][kInvN];
    const int i = threadIdx.x >> 5, j = threadIdx.x & 31;  // a warp per row
    double a = 0.0;
    const int x = i % 3, y = i / 3 % 3, z = i / 9, dx = j % 3 - x, dy = j / 3 % 3 - y, dz = j / 9 - z;
    if (j < kInvN && dx * dx <= 1 && dy * dy <= 1 && dz * dz <= 1)
        a = (double)coupling(c, cs, g, g.at(x, y, z), dx, dy, dz);
    for (int k = 0; k < kInvN; ++k) {
        double *row = pivot_row[k & 1], *column = pivot_column[k & 1];
        if (i == k) row[j] = a;
        if (j == k) column[i] = a;
        __syncthreads();
        const double inv_piv = 1.0 / row[k];
        const double r = j == k ? inv_piv : row[j] * inv_piv;  // row k / pivot
        a = i == k ? r : (j == k ? 0.0 : a) - column[i] * r;
    }
    if (j < kInvN) inv[i * kInvN + j] = a;
}

// ---- levels of side <= 9 in one block ---------------------------------------------
// The first level of side <= 9 and those below it (9, 5, 3) run in one block.
// Their operators do not change during a solve, so set-up writes them once
// into a compact image (pb_coarse27_image_f32): per level above the last, the
// 27 couplings of every node (offsets (dz, dy, dx) in lexicographic order, zero
// outside the grid; one coupling of all nodes after another), 1/diagonal and the
// prolongation weights; then the 3^3 inverse (FP64).
//
// A thread owns one node of one level, a level's threads its even nodes and then its
// odd ones (the colours), and keeps the node's couplings, weight, right-hand side and
// value in registers; the values go to shared memory split by colour, two copies of
// each, so that a colour's pass reads one copy and writes the other with one barrier,
// and its lanes read consecutive words.  Bound by latency: with the couplings in
// shared memory and two barriers a pass a cycle took 31 us.
constexpr int kC27N = 9;
constexpr int kC27Threads = 1024;
constexpr int kC27MaxLevels = 3;  // 9, 5, 3
constexpr int round32(int v) { return (v + 31) & ~31; }
static_assert(round32(9 * 9 * 9) + round32(5 * 5 * 5) + 27 <= kC27Threads, "one node per thread over all levels");

__host__ __device__ inline int round4(int v) { return (v + 3) & ~3; }

// Float offsets of the image sections.
struct CoarseLayout {
    int count;
    int n[kC27MaxLevels];
    int coef[kC27MaxLevels], invD[kC27MaxLevels], fac[kC27MaxLevels], inverse;
    int image;  // floats of the image (a multiple of 4)
};

__host__ __device__ inline CoarseLayout coarse_layout(int count, const int* sizes) {
    CoarseLayout c{};
    c.count = count;
    int off = 0;
    for (int l = 0; l < count; ++l) {
        const int n = sizes[l], N = n * n * n;
        c.n[l] = n;
        if (l == count - 1) break;  // the last level keeps its inverse only
        c.coef[l] = off;
        off += round4(27 * N);
        c.invD[l] = off;
        off += round4(N);
        c.fac[l] = off;
        off += round4(N);
    }
    c.inverse = off;  // 16-byte aligned: doubles
    off += round4(2 * kInvN * kInvN);
    c.image = off;
    return c;
}

__device__ __forceinline__ void unflatten(int i, int n, int& x, int& y, int& z) {
    x = i % n;
    y = (i / n) % n;
    z = i / (n * n);
}

// One node's couplings, 1/diagonal and weight into the image (set-up).
__global__ void coarse_image_kernel(const float* __restrict__ c, int64_t cs, Geom g, const float* __restrict__ invD,
                                    const float* __restrict__ fac, float* __restrict__ coef_out,
                                    float* __restrict__ invD_out, float* __restrict__ fac_out) {
    const int n = g.n, N = n * n * n;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    int x, y, z;
    unflatten(i, n, x, y, z);
    const int64_t p = g.at(x, y, z);
    int k = 0;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx, ++k)
                coef_out[(int64_t)k * N + i] = inside(x + dx, y + dy, z + dz, n) ? coupling(c, cs, g, p, dx, dy, dz) : 0.0f;
    invD_out[i] = invD[p];
    fac_out[i] = fac[p];
}

// A level's values in shared memory: the padded cube of side N + 2 (zero ghosts) by the
// parity of the linear index (a node's colour and its index's parity differ by one, so
// a colour is one parity), two copies.
template <int N>
struct Cube {
    static constexpr int M = N + 2, SIZE = M * M * M, HALF = (SIZE + 1) / 2;
    float e[2][2][HALF];  // by parity of the index, copy
    float res[SIZE];      // weighted residual, not split
    static __device__ __forceinline__ int at(int x, int y, int z) { return ((z + 1) * M + (y + 1)) * M + (x + 1); }
};

// What a thread holds of its node.
struct Node27 {
    int level = -1, x, y, z, c, colour;  // c: index in the padded cube
    float a[27], inv, fac, rhs, e;
};

// sum over the 26 neighbours, and the node itself where CENTRE, of a_K e[J + K] in the couplings' order.
template <int N, bool CENTRE>
__device__ __forceinline__ float stencil_cube(const Cube<N>& cube, const Node27& v, const int (&copy)[2]) {
    constexpr int M = Cube<N>::M;
    const int odd = v.c & 1;
    const float* same = &cube.e[odd][copy[odd]][v.c >> 1];
    const float* other = &cube.e[odd ^ 1][copy[odd ^ 1]][(v.c >> 1) + odd];
    float s = 0.0f;
    int k = 0;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx, ++k) {
                const int d = dx + dy * M + dz * M * M;
                if (d == 0) {
                    if (CENTRE) s += v.a[k] * v.e;
                } else {
                    s += v.a[k] * ((d & 1) ? other[(d - 1) / 2] : same[d / 2]);
                }
            }
    return s;
}

// Red-black ordered sweeps: a colour's new values come from the current iterate (its own
// colour's neighbours included) and go to its other copy, as the multi-block colour
// passes do.  Every thread of the block calls it; from_zero: e is zero.
template <int N>
__device__ __forceinline__ void cube_relax(Cube<N>& cube, Node27& v, int level, int (&copy)[2], int iters,
                                           bool from_zero) {
    for (int pass = 0; pass < 2 * iters; ++pass) {
        const int colour = pass & 1, parity = colour ^ 1;
        if (v.level == level && v.colour == colour) {
            const float s = from_zero && pass == 0 ? 0.0f : stencil_cube<N, false>(cube, v, copy);
            v.e = (v.rhs - s) * v.inv;
            cube.e[parity][copy[parity] ^ 1][v.c >> 1] = v.e;
        }
        copy[parity] ^= 1;
        __syncthreads();
    }
}

template <int N>
__device__ __forceinline__ void cube_residual(Cube<N>& cube, const Node27& v, int level, const int (&copy)[2]) {
    if (v.level == level) cube.res[v.c] = v.fac * (v.rhs - stencil_cube<N, true>(cube, v, copy));
    __syncthreads();
}

// The restricted residual at coarse node (x, y, z).
template <int N>
__device__ __forceinline__ float cube_restrict(const Cube<N>& cube, int x, int y, int z) {
    constexpr int M = Cube<N>::M;
    const float* r = cube.res + Cube<N>::at(2 * x, 2 * y, 2 * z);
    float s = 0.0f;
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx)
                s += r[dx + dy * M + dz * M * M] * (float)((dx ? 1 : 2) * (dy ? 1 : 2) * (dz ? 1 : 2));
    return s * (1.0f / 64.0f);
}

// e += weight * trilinear coarse correction, the mean of the 8 corners (a corner repeated
// on even axes); value(x, y, z): the coarse level's.
template <int N, typename Value>
__device__ __forceinline__ void cube_prolong(Cube<N>& cube, Node27& v, int level, const int (&copy)[2], Value value) {
    if (v.level == level) {
        const int x0 = v.x >> 1, y0 = v.y >> 1, z0 = v.z >> 1;
        const int x1 = x0 + (v.x & 1), y1 = y0 + (v.y & 1), z1 = z0 + (v.z & 1);
        v.e += v.fac * (0.125f * (value(x0, y0, z0) + value(x1, y0, z0) + value(x0, y1, z0) + value(x1, y1, z0) +
                                  value(x0, y0, z1) + value(x1, y0, z1) + value(x0, y1, z1) + value(x1, y1, z1)));
        const int odd = v.c & 1;
        cube.e[odd][copy[odd]][v.c >> 1] = v.e;
    }
    __syncthreads();
}

// V(pre, post) on the first level and `inner` sweeps each way on the one between; sides (9, 5, 3), (5, 3) or (3).
__device__ __forceinline__ void coarse27_body(const float* __restrict__ image, const CoarseLayout& lay,
                                              const float* __restrict__ rhs0, float* __restrict__ e0, Geom g0,
                                              int pre, int post, int inner) {
    __shared__ struct {
        Cube<9> nine;
        Cube<5> five;
    } cubes;
    __shared__ double inverse[kInvN * kInvN], rhs3[kInvN];
    __shared__ float e3[kInvN];
    const int tid = threadIdx.x;
    for (int i = tid; i < (int)(sizeof(cubes) / sizeof(float)); i += kC27Threads) reinterpret_cast<float*>(&cubes)[i] = 0.0f;
    if (tid < kInvN * kInvN) inverse[tid] = reinterpret_cast<const double*>(image + lay.inverse)[tid];
    Node27 v;
    int first = 0;  // the level's first thread; the last level's 27 threads come after the others
#pragma unroll
    for (int l = 0; l < kC27MaxLevels; ++l) {
        if (l >= lay.count) break;
        const int n = lay.n[l], count = n * n * n, t = tid - first;
        if (t >= 0 && t < count) {
            v.level = l;
            const int even = (count + 1) / 2;
            const int i = l + 1 == lay.count ? t : t < even ? 2 * t : 2 * (t - even) + 1;
            unflatten(i, n, v.x, v.y, v.z);
            v.colour = (v.x + v.y + v.z) & 1;
            v.c = ((v.z + 1) * (n + 2) + (v.y + 1)) * (n + 2) + (v.x + 1);
            v.e = 0.0f;
            if (l == 0) v.rhs = rhs0[g0.at(v.x, v.y, v.z)];
            if (l + 1 < lay.count) {
#pragma unroll
                for (int k = 0; k < 27; ++k) v.a[k] = image[lay.coef[l] + k * count + i];
                v.inv = image[lay.invD[l] + i];
                v.fac = image[lay.fac[l] + i];
            }
        }
        first += round32(count);
    }
    __syncthreads();
    const int last = lay.count - 1;
    int copy9[2] = {0, 0}, copy5[2] = {0, 0};
    if (lay.n[0] == 9) {
        cube_relax<9>(cubes.nine, v, 0, copy9, pre, true);
        cube_residual<9>(cubes.nine, v, 0, copy9);
        if (v.level == 1) v.rhs = cube_restrict<9>(cubes.nine, v.x, v.y, v.z);
    }
    const int level5 = lay.count - 2;  // -1: none
    if (level5 >= 0) {
        cube_relax<5>(cubes.five, v, level5, copy5, level5 == 0 ? pre : inner, true);
        cube_residual<5>(cubes.five, v, level5, copy5);
        if (v.level == last) v.rhs = cube_restrict<5>(cubes.five, v.x, v.y, v.z);
    }
    const int own3 = (v.z * 3 + v.y) * 3 + v.x;
    if (v.level == last) rhs3[own3] = (double)v.rhs;
    __syncthreads();
    if (v.level == last) {  // side 3: e = A^-1 rhs
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < kInvN; ++j) sum += inverse[own3 * kInvN + j] * rhs3[j];
        e3[own3] = v.e = (float)sum;
    }
    __syncthreads();
    if (level5 >= 0) {
        cube_prolong<5>(cubes.five, v, level5, copy5, [&](int x, int y, int z) { return e3[(z * 3 + y) * 3 + x]; });
        cube_relax<5>(cubes.five, v, level5, copy5, level5 == 0 ? post : inner, false);
    }
    if (lay.n[0] == 9) {
        cube_prolong<9>(cubes.nine, v, 0, copy9, [&](int x, int y, int z) {
            const int c = Cube<5>::at(x, y, z);
            return cubes.five.e[c & 1][copy5[c & 1]][c >> 1];
        });
        cube_relax<9>(cubes.nine, v, 0, copy9, post, false);
    }
    if (v.level == 0) e0[g0.at(v.x, v.y, v.z)] = v.e;
}

__global__ void __launch_bounds__(kC27Threads) coarse27_kernel(const float* __restrict__ image, CoarseLayout lay,
                                                               const float* __restrict__ rhs0,
                                                               float* __restrict__ e0, Geom g0, int pre, int post,
                                                               int inner) {
    coarse27_body(image, lay, rhs0, e0, g0, pre, post, inner);
}

// ---- grouped launches (batch.cuh) ----------------------------------------------------

// relax27p: ptr[0] e_prev (null: from zero), ptr[1] e_next, ptr[2] rhs, ptr[3] h0, ptr[4] h1, ptr[5] inv0,
// ptr[6] inv1.  Colour COLOUR of every grid.
template <int COLOUR, bool ZERO>
__global__ void __launch_bounds__(256) relax27p_grouped_kernel(const batch::GridDesc* __restrict__ descs, int count,
                                                               const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    const int n = (int)d.n;
    relax27p_body<COLOUR, ZERO>((const float*)d.ptr[0], (float*)d.ptr[1], (const float*)d.ptr[2],
                                (const __half*)d.ptr[3 + COLOUR], (const float*)d.ptr[5 + COLOUR], geom(n),
                                packed_of(n), bx, by);
}

// residual27p: ptr[0] e, ptr[1] rhs, ptr[2] h0, ptr[3] h1, ptr[4] inv0, ptr[5] inv1, ptr[6] weights, ptr[7] res.
__global__ void __launch_bounds__(256) residual27p_grouped_kernel(const batch::GridDesc* __restrict__ descs,
                                                                  int count, const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    const int n = (int)d.n;
    residual27p_body((const float*)d.ptr[0], (const float*)d.ptr[1], (const __half*)d.ptr[2],
                     (const __half*)d.ptr[3], (const float*)d.ptr[4], (const float*)d.ptr[5], (const float*)d.ptr[6],
                     geom(n), packed_of(n), (float*)d.ptr[7], bx, by);
}

// restrict27: ptr[0] fine residual, ptr[1] coarse rhs; d.n is the fine side.
__global__ void __launch_bounds__(256) restrict27_grouped_kernel(const batch::GridDesc* __restrict__ descs, int count,
                                                                 const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    const int n = (int)d.n;
    restrict27_body((const float*)d.ptr[0], geom(n), (float*)d.ptr[1], geom((n + 1) / 2), bx, by);
}

// coarse27: one block per cloud; ptr[0] image, ptr[1] rhs, ptr[2] e; d.n the first level's side (9, 5 or 3
// levels below it); aux[0..2] pre, post, inner.  Every grid of one launch has the same side.
__global__ void __launch_bounds__(kC27Threads) coarse27_grouped_kernel(const batch::GridDesc* __restrict__ descs,
                                                                       int count, const int* __restrict__ flags,
                                                                       CoarseLayout lay) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    coarse27_body((const float*)d.ptr[0], lay, (const float*)d.ptr[1], (float*)d.ptr[2], geom((int)d.n),
                  (int)d.aux[0], (int)d.aux[1], (int)d.aux[2]);
}


}  // namespace pb

using namespace pb;

static bool level_side_ok(int64_t n) { return n >= 3 && n <= 4097 && ((n - 1) & (n - 2)) == 0; }

// Scratch floats of the separable product for a slab of kp coarse planes:
// stage x (cn x fn x nz) and stage y (cn x cn x nz), 27 planes each, nz =
// 2 kp + 1 fine planes.
static int64_t galerkin_slab_floats(int fn, int kp) {
    const int cn = (fn + 1) / 2;
    const int64_t nz = 2 * (int64_t)kp + 1;
    return 27 * ((int64_t)cn * fn + (int64_t)cn * cn) * nz;
}

// Scratch bytes for the whole level in one slab (any size down to one coarse
// plane, galerkin_slab_floats(fn, 1) * 4 bytes, works in more slabs); 0 for
// a 7-point fine level.
extern "C" size_t pb_galerkin_workspace_size(int64_t fine_n, int fine_is_7pt) {
    if (!level_side_ok(fine_n) || fine_is_7pt) return 0;
    return (size_t)galerkin_slab_floats((int)fine_n, (int)((fine_n + 1) / 2)) * sizeof(float) + 256;
}

// Coarse 27-point operator (14 planes, plane stride padded_size(cn)) of the
// level below a fine level of side fine_n with prolongation weights
// fine_weights.  fine_is_7pt: `fine` is the level-0 diagonal D (couplings
// -(n-1)^2, direct sum, no scratch); otherwise `fine` holds 14 planes and the
// separable stages run over slabs of coarse planes that fit the workspace.
// occupancy: the words of the screen behind a 7-point level (pb_refine_start_sparse_f64), or null.
extern "C" int pb_galerkin_sparse_f32(const float* fine, int64_t fine_n, int fine_is_7pt, const float* fine_weights,
                                      const void* occupancy, float* coarse, void* workspace, size_t workspace_bytes,
                                      void* stream) {
    if (!level_side_ok(fine_n) || !fine || !coarse || !fine_weights) return fail(PB_ERR_INVALID, "galerkin: bad args");
    const int fn = (int)fine_n, cn = (fn + 1) / 2;
    const Geom gf = geom(fn), gc = geom(cn);
    cudaStream_t s = (cudaStream_t)stream;
    if (fine_is_7pt) {
        const float h2 = (float)(fn - 1) * (float)(fn - 1);
        galerkin7_kernel<<<plane_grid(cn, 128), 128, 0, s>>>(fine, fine_weights, screen_map(occupancy), Plain14(h2), gf,
                                                             h2, coarse, padded_size(cn), gc);
        PB_CHECK_LAUNCH("galerkin7_kernel");
        return PB_OK;
    }
    const int64_t have = workspace ? (int64_t)(workspace_bytes / sizeof(float)) : 0;
    if (have < galerkin_slab_floats(fn, 1))
        return fail(PB_ERR_WORKSPACE, "galerkin: workspace needs at least %lld bytes",
                    (long long)(galerkin_slab_floats(fn, 1) * (int64_t)sizeof(float)));
    if (cn <= kSmallCoarse) {
        galerkin_small_kernel<<<blocks_for((int64_t)cn * cn * cn, 4), 128, 0, s>>>(fine, padded_size(fn), fine_weights, gf,
                                                                                coarse, padded_size(cn), gc);
        PB_CHECK_LAUNCH("galerkin_small_kernel");
        return PB_OK;
    }
    int kp = cn;
    while (kp > 1 && galerkin_slab_floats(fn, kp) > have) kp = (kp + 1) / 2;
    float* bx = static_cast<float*>(workspace);
    for (int k0 = 0; k0 < cn; k0 += kp) {
        const int k1 = min(cn, k0 + kp);
        const int zlo = max(0, 2 * k0 - 1), zhi = min(fn, 2 * k1);
        const int nz = zhi - zlo;
        const int64_t px = (int64_t)cn * fn * nz, py = (int64_t)cn * cn * nz;
        float* by = bx + 27 * px;
        galerkin_x_kernel<<<dim3((cn * fn + 127) / 128, nz), 128, 0, s>>>(fine, padded_size(fn), fine_weights, gf,
                                                                          cn, zlo, bx, px);
        PB_CHECK_LAUNCH("galerkin_x_kernel");
        galerkin_y_kernel<<<dim3((cn * cn + 127) / 128, nz), 128, 0, s>>>(bx, px, fn, cn, by, py);
        PB_CHECK_LAUNCH("galerkin_y_kernel");
        galerkin_z_kernel<<<dim3((cn * cn + 127) / 128, k1 - k0), 128, 0, s>>>(by, py, fn, zlo, k0, coarse,
                                                                              padded_size(cn), gc);
        PB_CHECK_LAUNCH("galerkin_z_kernel");
    }
    return PB_OK;
}

extern "C" int pb_galerkin_f32(const float* fine, int64_t fine_n, int fine_is_7pt, const float* fine_weights,
                               float* coarse, void* workspace, size_t workspace_bytes, void* stream) {
    return pb_galerkin_sparse_f32(fine, fine_n, fine_is_7pt, fine_weights, nullptr, coarse, workspace, workspace_bytes,
                                  stream);
}

// 14 planes of a 7-point level (diagonal D, off-diagonals -(n-1)^2).
extern "C" int pb_level27_from7_f32(const float* D, int64_t n, float* coef, void* stream) {
    if (!level_side_ok(n) || !D || !coef) return fail(PB_ERR_INVALID, "level27 from 7: bad args");
    level7_to_27_kernel<<<plane_grid((int)n, 128), 128, 0, (cudaStream_t)stream>>>(
        D, geom((int)n), (float)(n - 1) * (float)(n - 1), coef, padded_size((int)n));
    PB_CHECK_LAUNCH("level7_to_27_kernel");
    return PB_OK;
}

// invD = 1 / diagonal and the prolongation weights of a 27-point level.
extern "C" int pb_level27_finish_f32(const float* coef, int64_t n, float* invD, float* weights, void* stream) {
    if (!level_side_ok(n) || !coef || !invD || !weights) return fail(PB_ERR_INVALID, "level27 finish: bad args");
    level27_finish_kernel<<<plane_grid((int)n, 128), 128, 0, (cudaStream_t)stream>>>(
        coef, padded_size((int)n), geom((int)n), invD, weights);
    PB_CHECK_LAUNCH("level27_finish_kernel");
    return PB_OK;
}

// Inverse (27 x 27, FP32 row-major) of a 27-point level of side 3.
extern "C" int pb_coarse_inverse_f64(const float* coef, int64_t n, double* inverse, void* stream) {
    if (n != 3 || !coef || !inverse) return fail(PB_ERR_INVALID, "coarse inverse: side must be 3");
    coarse_inverse_kernel<<<1, 32 * kInvN, 0, (cudaStream_t)stream>>>(coef, padded_size(3), geom(3), inverse);
    PB_CHECK_LAUNCH("coarse_inverse_kernel");
    return PB_OK;
}

static int coarse_sizes(int64_t count, const int64_t* sizes, int* out) {
    if (count < 1 || count > kC27MaxLevels || !sizes) return fail(PB_ERR_INVALID, "coarse27: 1 to 3 levels");
    for (int l = 0; l < count; ++l) {
        if (!level_side_ok(sizes[l]) || sizes[l] > kC27N || (l && sizes[l] != (sizes[l - 1] + 1) / 2))
            return fail(PB_ERR_INVALID, "coarse27: level sides must halve from <= 9 down to 3");
        out[l] = (int)sizes[l];
    }
    if (sizes[count - 1] != 3) return fail(PB_ERR_INVALID, "coarse27: the last level must have side 3");
    return PB_OK;
}

// Bytes of the image of levels `sizes` (finest first, side <= 9 halving to 3).
extern "C" size_t pb_coarse27_image_size(int64_t count, const int64_t* sizes) {
    int sz[kC27MaxLevels];
    if (coarse_sizes(count, sizes, sz) != PB_OK) return 0;
    return (size_t)coarse_layout((int)count, sz).image * sizeof(float);
}

// The image the single-block cycle reads: per level but the last, couplings
// (from its 14 planes), 1/diagonal and prolongation weights; then the 3^3
// inverse (FP64, from pb_coarse_inverse_f64).  image: 16-byte aligned.
extern "C" int pb_coarse27_image_f32(int64_t count, const int64_t* sizes, const float* const* coef,
                                     const float* const* invD, const float* const* weights, const double* inverse,
                                     float* image, size_t image_bytes, void* stream) {
    int sz[kC27MaxLevels];
    PB_TRY(coarse_sizes(count, sizes, sz));
    if (!coef || !invD || !weights || !inverse || !image || (reinterpret_cast<uintptr_t>(image) & 15))
        return fail(PB_ERR_INVALID, "coarse27 image: bad args");
    const CoarseLayout lay = coarse_layout((int)count, sz);
    if (image_bytes < (size_t)lay.image * sizeof(float)) return fail(PB_ERR_WORKSPACE, "coarse27 image: too small");
    cudaStream_t s = (cudaStream_t)stream;
    for (int l = 0; l + 1 < count; ++l) {
        if (!coef[l] || !invD[l] || !weights[l]) return fail(PB_ERR_INVALID, "coarse27 image: null level array");
        const int N = sz[l] * sz[l] * sz[l];
        coarse_image_kernel<<<(N + 255) / 256, 256, 0, s>>>(coef[l], padded_size(sz[l]), geom(sz[l]), invD[l],
                                                            weights[l], image + lay.coef[l], image + lay.invD[l],
                                                            image + lay.fac[l]);
        PB_CHECK_LAUNCH("coarse_image_kernel");
    }
    PB_CHECK_CUDA(cudaMemcpyAsync(image + lay.inverse, inverse, sizeof(double) * kInvN * kInvN,
                                  cudaMemcpyDeviceToDevice, s),
                  "coarse27 image inverse");
    return PB_OK;
}

// Levels of side <= 9 in one block from their image: V(pre, post) on the
// first, `inner` sweeps each way on the others, the last (side 3) solved with
// its inverse.  rhs: the first level's right-hand side (padded layout); e
// receives its correction (padded layout; ghosts untouched).
extern "C" int pb_coarse27_cycle_f32(int64_t count, const int64_t* sizes, const float* image, const float* rhs,
                                     float* e, int64_t pre, int64_t post, int64_t inner, void* stream) {
    int sz[kC27MaxLevels];
    PB_TRY(coarse_sizes(count, sizes, sz));
    if (!image || !rhs || !e || (reinterpret_cast<uintptr_t>(image) & 15))
        return fail(PB_ERR_INVALID, "coarse27 cycle: bad args");
    if (pre < 0 || post < 0 || inner < 0 || pre > 64 || post > 64 || inner > 64)
        return fail(PB_ERR_INVALID, "coarse27 cycle: sweep counts must be in [0, 64]");
    const CoarseLayout lay = coarse_layout((int)count, sz);
    coarse27_kernel<<<1, kC27Threads, 0, (cudaStream_t)stream>>>(image, lay, rhs, e, geom(sz[0]), (int)pre, (int)post,
                                                                  (int)inner);
    PB_CHECK_LAUNCH("coarse27_kernel");
    return PB_OK;
}

// ---- packed levels ----------------------------------------------------------------
// Bytes of one colour's packed couplings (32 FP16 per node) and of its 1/diagonal.
extern "C" int pb_packed27_size(int64_t n, int64_t* coupling_bytes, int64_t* inverse_bytes) {
    if (!level_side_ok(n)) return fail(PB_ERR_INVALID, "packed27 size: bad side");
    const Packed pk = packed_of((int)n);
    if (coupling_bytes) *coupling_bytes = kPackedStride * pk.cs * (int64_t)sizeof(__half);
    if (inverse_bytes) *inverse_bytes = pk.cs * (int64_t)sizeof(float);
    return PB_OK;
}

// Packs a 27-point level (14 planes): per colour c, couplings h_c and 1/diagonal inv_c.
extern "C" int pb_pack27_f32(const float* coef, int64_t n, void* h0, void* h1, float* inv0, float* inv1,
                             void* stream) {
    if (!level_side_ok(n) || !coef || !h0 || !h1 || !inv0 || !inv1) return fail(PB_ERR_INVALID, "pack27: bad args");
    pack27_kernel<<<plane_grid((int)n, 256), 256, 0, (cudaStream_t)stream>>>(
        coef, padded_size((int)n), geom((int)n), packed_of((int)n), (__half*)h0, (__half*)h1, inv0, inv1);
    PB_CHECK_LAUNCH("pack27_kernel");
    return PB_OK;
}

// One red-black ordered sweep e_next <- S(e_prev) on a packed level (e_prev null: from zero).
extern "C" int pb_relax27p_f32(const float* e_prev, float* e_next, const float* rhs, const void* h0, const void* h1,
                               const float* inv0, const float* inv1, int64_t n, void* stream) {
    if (!level_side_ok(n) || !e_next || !rhs || !h0 || !h1 || !inv0 || !inv1 || e_prev == e_next)
        return fail(PB_ERR_INVALID, "relax27p: bad args");
    cudaStream_t s = (cudaStream_t)stream;
    const Geom g = geom((int)n);
    const Packed pk = packed_of((int)n);
    const dim3 block(256);
    const dim3 grid((pk.Pc * (int)n + 255) / 256, (int)n);
    const __half *a = (const __half*)h0, *b = (const __half*)h1;
    if (tuned(PB_TUNE_RELAX27_VARIANT, n, 0) == 1) {  // shared-memory staged neighbours
        const int tiles = ((pk.Pc + kTPi - 1) / kTPi) * (((int)n + kTPy - 1) / kTPy);
        const int64_t want = 2LL * 8 * kSMs;  // about two waves of 8 resident blocks per SM
        int tz = (int)(((int64_t)n * tiles + want - 1) / want);
        tz = tz < 2 ? 2 : (tz > 16 ? 16 : tz);
        const dim3 tg((pk.Pc + kTPi - 1) / kTPi, ((int)n + kTPy - 1) / kTPy, ((int)n + tz - 1) / tz);
        if (e_prev) {
            relax27p_tiled_kernel<0, false><<<tg, kTPi * kTPy, 0, s>>>(e_prev, e_next, rhs, a, inv0, g, pk, tz);
            PB_CHECK_LAUNCH("relax27p_tiled_kernel");
            relax27p_tiled_kernel<1, false><<<tg, kTPi * kTPy, 0, s>>>(e_prev, e_next, rhs, b, inv1, g, pk, tz);
        } else {
            relax27p_kernel<0, true><<<grid, block, 0, s>>>(nullptr, e_next, rhs, a, inv0, g, pk);  // no neighbours
            PB_CHECK_LAUNCH("relax27p_kernel");
            relax27p_tiled_kernel<1, true><<<tg, kTPi * kTPy, 0, s>>>(nullptr, e_next, rhs, b, inv1, g, pk, tz);
        }
        PB_CHECK_LAUNCH("relax27p_tiled_kernel");
        return PB_OK;
    }
    if (e_prev) {
        relax27p_kernel<0, false><<<grid, block, 0, s>>>(e_prev, e_next, rhs, a, inv0, g, pk);
        PB_CHECK_LAUNCH("relax27p_kernel");
        relax27p_kernel<1, false><<<grid, block, 0, s>>>(e_prev, e_next, rhs, b, inv1, g, pk);
    } else {
        relax27p_kernel<0, true><<<grid, block, 0, s>>>(nullptr, e_next, rhs, a, inv0, g, pk);
        PB_CHECK_LAUNCH("relax27p_kernel");
        relax27p_kernel<1, true><<<grid, block, 0, s>>>(nullptr, e_next, rhs, b, inv1, g, pk);
    }
    PB_CHECK_LAUNCH("relax27p_kernel");
    return PB_OK;
}

// res = weights * (rhs - A e) with the packed operator, then coarse_rhs = P^T res / 8.
extern "C" int pb_residual_restrict27p_f32(const float* e, const float* rhs, const void* h0, const void* h1,
                                           const float* inv0, const float* inv1, const float* weights, int64_t n,
                                           float* res, float* coarse_rhs, void* stream) {
    if (!level_side_ok(n) || n < 5 || !e || !rhs || !h0 || !h1 || !inv0 || !inv1 || !weights || !res || !coarse_rhs)
        return fail(PB_ERR_INVALID, "residual_restrict27p: bad args");
    cudaStream_t s = (cudaStream_t)stream;
    const int fn = (int)n, cn = (fn + 1) / 2;
    if (tuned(PB_TUNE_RESIDUAL27_VARIANT, n, 0) == 1) {  // shared-memory staged e planes
        const int tiles = ((fn + kTRx - 1) / kTRx) * ((fn + kTRy - 1) / kTRy);
        const int64_t want = 2LL * 8 * kSMs;
        int tz = (int)(((int64_t)fn * tiles + want - 1) / want);
        tz = tz < 2 ? 2 : (tz > 16 ? 16 : tz);
        const dim3 tg((fn + kTRx - 1) / kTRx, (fn + kTRy - 1) / kTRy, (fn + tz - 1) / tz);
        residual27p_tiled_kernel<<<tg, kTRx * kTRy, 0, s>>>(e, rhs, (const __half*)h0, (const __half*)h1, inv0, inv1,
                                                           weights, geom(fn), packed_of(fn), res, tz);
        PB_CHECK_LAUNCH("residual27p_tiled_kernel");
    } else {
        residual27p_kernel<<<dim3((fn * fn + 255) / 256, fn), 256, 0, s>>>(
            e, rhs, (const __half*)h0, (const __half*)h1, inv0, inv1, weights, geom(fn), packed_of(fn), res);
        PB_CHECK_LAUNCH("residual27p_kernel");
    }
    restrict27_kernel<<<plane_grid(cn, 256), 256, 0, s>>>(res, geom(fn), coarse_rhs, geom(cn));
    PB_CHECK_LAUNCH("restrict27_kernel");
    return PB_OK;
}

// ---- grouped launches (batch.cuh) ----------------------------------------------------

namespace pb {
namespace batch {

int describe_relax27p(GridDesc& d, bool zero) {
    const int n = (int)d.n;
    if (!level_side_ok(n) || (!zero && !d.ptr[0]) || !d.ptr[1] || !d.ptr[2] || !d.ptr[3] || !d.ptr[4] || !d.ptr[5] ||
        !d.ptr[6] || d.ptr[0] == d.ptr[1])
        return fail(PB_ERR_INVALID, "batch relax27p: bad args");
    const Packed pk = packed_of(n);
    d.gx = (pk.Pc * n + 255) / 256;
    d.gy = n;
    d.gz = 1;
    return PB_OK;
}

int launch_relax27p(const GridDesc* descs, int count, int64_t blocks, bool zero, const int* flags, cudaStream_t s) {
    if (zero) {
        relax27p_grouped_kernel<0, true><<<(unsigned)blocks, 256, 0, s>>>(descs, count, flags);
        PB_CHECK_LAUNCH("relax27p_grouped_kernel");
        relax27p_grouped_kernel<1, true><<<(unsigned)blocks, 256, 0, s>>>(descs, count, flags);
    } else {
        relax27p_grouped_kernel<0, false><<<(unsigned)blocks, 256, 0, s>>>(descs, count, flags);
        PB_CHECK_LAUNCH("relax27p_grouped_kernel");
        relax27p_grouped_kernel<1, false><<<(unsigned)blocks, 256, 0, s>>>(descs, count, flags);
    }
    PB_CHECK_LAUNCH("relax27p_grouped_kernel");
    return PB_OK;
}

int describe_residual27p(GridDesc& d) {
    const int n = (int)d.n;
    for (int k = 0; k < 8; ++k)
        if (!d.ptr[k]) return fail(PB_ERR_INVALID, "batch residual27p: bad args");
    if (!level_side_ok(n) || n < 5) return fail(PB_ERR_INVALID, "batch residual27p: bad side");
    d.gx = (n * n + 255) / 256;
    d.gy = n;
    d.gz = 1;
    return PB_OK;
}

int launch_residual27p(const GridDesc* descs, int count, int64_t blocks, const int* flags, cudaStream_t s) {
    residual27p_grouped_kernel<<<(unsigned)blocks, 256, 0, s>>>(descs, count, flags);
    PB_CHECK_LAUNCH("residual27p_grouped_kernel");
    return PB_OK;
}

int describe_restrict27(GridDesc& d) {
    const int n = (int)d.n;
    if (!level_side_ok(n) || n < 5 || !d.ptr[0] || !d.ptr[1]) return fail(PB_ERR_INVALID, "batch restrict27: bad args");
    const int cn = (n + 1) / 2;
    d.gx = (cn * cn + 255) / 256;
    d.gy = cn;
    d.gz = 1;
    return PB_OK;
}

int launch_restrict27(const GridDesc* descs, int count, int64_t blocks, const int* flags, cudaStream_t s) {
    restrict27_grouped_kernel<<<(unsigned)blocks, 256, 0, s>>>(descs, count, flags);
    PB_CHECK_LAUNCH("restrict27_grouped_kernel");
    return PB_OK;
}

int describe_coarse27(GridDesc& d) {
    const int n = (int)d.n;
    if (!level_side_ok(n) || n > kC27N || !d.ptr[0] || !d.ptr[1] || !d.ptr[2] ||
        (reinterpret_cast<uintptr_t>(d.ptr[0]) & 15))
        return fail(PB_ERR_INVALID, "batch coarse27: bad args");
    if (d.aux[0] < 0 || d.aux[1] < 0 || d.aux[2] < 0 || d.aux[0] > 64 || d.aux[1] > 64 || d.aux[2] > 64)
        return fail(PB_ERR_INVALID, "batch coarse27: sweep counts must be in [0, 64]");
    d.gx = d.gy = d.gz = 1;
    return PB_OK;
}

int launch_coarse27(const GridDesc* descs, int count, int64_t blocks, int first_side, const int* flags,
                    cudaStream_t s) {
    int sz[kC27MaxLevels];
    int levels = 0;
    for (int m = first_side; levels < kC27MaxLevels; m = (m + 1) / 2) {
        sz[levels++] = m;
        if (m == 3) break;
    }
    if (sz[levels - 1] != 3) return fail(PB_ERR_INVALID, "batch coarse27: first side must be 9, 5 or 3");
    const CoarseLayout lay = coarse_layout(levels, sz);
    coarse27_grouped_kernel<<<(unsigned)blocks, kC27Threads, 0, s>>>(descs, count, flags, lay);
    PB_CHECK_LAUNCH("coarse27_grouped_kernel");
    return PB_OK;
}

}  // namespace batch
}  // namespace pb

// ---- a whole hierarchy's set-up in one call ---------------------------------------
// The sequence Hierarchy32.setup issues level by level, from one host call:
// level 0 from the screen, each coarser level's Galerkin operator from the one
// above, finish, and the packing of every packed level right after the product
// that reads it for the last time; then the 3^3 inverse and the coarse image.
// Same launches in the same order as the separate entry points.
// occupancy: the words of level 0's screen where pb_refine_start_sparse_f64 wrote both (null: none).
extern "C" int pb_hierarchy_setup_sparse_f32(int64_t levels, const int64_t* sides, const void* const* arrays,
                                             int64_t first_coarse, const double* screen, double point_weight,
                                             const void* occupancy, void* galerkin_ws, size_t galerkin_bytes,
                                             double* inverse, float* image, size_t image_bytes, void* stream) {
    constexpr int A = PB_LEVEL_ARRAYS;
    if (levels < 2 || levels > 13 || !sides || !arrays || !inverse || !image || first_coarse < 0 ||
        first_coarse >= levels)
        return fail(PB_ERR_INVALID, "hierarchy setup: bad args");
    for (int64_t l = 0; l < levels; ++l) {
        if (!level_side_ok(sides[l]) || (l && sides[l] != (sides[l - 1] + 1) / 2))
            return fail(PB_ERR_INVALID, "hierarchy setup: level sides must halve from a 2^k + 1 side down to 3");
        if (!arrays[l * A + 1] || !arrays[l * A + 2] || (l && !arrays[l * A + 3]))
            return fail(PB_ERR_INVALID, "hierarchy setup: level %lld misses invD, weights or coef", (long long)l);
    }
    if (sides[levels - 1] != 3) return fail(PB_ERR_INVALID, "hierarchy setup: the last level must have side 3");
    auto D = [&](int64_t l) { return (float*)arrays[l * A + 0]; };
    auto invD = [&](int64_t l) { return (float*)arrays[l * A + 1]; };
    auto W = [&](int64_t l) { return (float*)arrays[l * A + 2]; };
    auto coef = [&](int64_t l) { return (float*)arrays[l * A + 3]; };
    auto packed = [&](int64_t l) { return arrays[l * A + 4] != nullptr; };
    const bool seven = coef(0) == nullptr;
    if (!D(0)) return fail(PB_ERR_INVALID, "hierarchy setup: level 0 needs D");
    if (seven && first_coarse == 0)
        return fail(PB_ERR_INVALID, "hierarchy setup: a 7-point level 0 cannot be part of the coarse cycle");
    // without a screen level 0's D, 1/D and weights are there already (pb_refine_start_f64)
    if (screen) PB_TRY(pb_level_setup_f32(screen, sides[0], point_weight, D(0), invD(0), W(0), stream));
    if (!seven) {
        PB_TRY(pb_level27_from7_f32(D(0), sides[0], coef(0), stream));
        PB_TRY(pb_level27_finish_f32(coef(0), sides[0], invD(0), W(0), stream));
    }
    for (int64_t l = 1; l < levels; ++l) {
        const bool fine7 = l == 1 && seven;
        PB_TRY(pb_galerkin_sparse_f32(fine7 ? D(0) : coef(l - 1), sides[l - 1], fine7 ? 1 : 0, W(l - 1), occupancy,
                                      coef(l), galerkin_ws, galerkin_bytes, stream));
        PB_TRY(pb_level27_finish_f32(coef(l), sides[l], invD(l), W(l), stream));
        if (packed(l - 1))
            PB_TRY(pb_pack27_f32(coef(l - 1), sides[l - 1], (void*)arrays[(l - 1) * A + 4],
                                 (void*)arrays[(l - 1) * A + 5], (float*)arrays[(l - 1) * A + 6],
                                 (float*)arrays[(l - 1) * A + 7], stream));
    }
    PB_TRY(pb_coarse_inverse_f64(coef(levels - 1), 3, inverse, stream));
    const int64_t tail = levels - first_coarse;
    const float* tc[kC27MaxLevels];
    const float* ti[kC27MaxLevels];
    const float* tw[kC27MaxLevels];
    if (tail < 1 || tail > kC27MaxLevels) return fail(PB_ERR_INVALID, "hierarchy setup: 1 to 3 levels of side <= 9");
    for (int64_t k = 0; k < tail; ++k) {
        tc[k] = coef(first_coarse + k);
        ti[k] = invD(first_coarse + k);
        tw[k] = W(first_coarse + k);
    }
    return pb_coarse27_image_f32(tail, sides + first_coarse, tc, ti, tw, inverse, image, image_bytes, stream);
}

extern "C" int pb_hierarchy_setup_f32(int64_t levels, const int64_t* sides, const void* const* arrays,
                                      int64_t first_coarse, const double* screen, double point_weight,
                                      void* galerkin_ws, size_t galerkin_bytes, double* inverse, float* image,
                                      size_t image_bytes, void* stream) {
    if (!screen) return fail(PB_ERR_INVALID, "hierarchy setup: null screen");
    return pb_hierarchy_setup_sparse_f32(levels, sides, arrays, first_coarse, screen, point_weight, nullptr, galerkin_ws,
                                         galerkin_bytes, inverse, image, image_bytes, stream);
}
