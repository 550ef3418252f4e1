// FP64 flexible conjugate gradients, FCG(1), around the FP32 V-cycle.
//
// The reference solves A x = b by repeating V-cycles (python/mojo_poissonrecon/
// core.py:274-285).  Used as a preconditioner z = M(r) inside a Krylov loop
// the V-cycle needs fewer applications.  Because M is an FP32 V-cycle (not a
// fixed symmetric operator), the flexible form is used: each direction is
// A-orthogonalised against the previous one only.
//
//   r = b - A x;  repeat:  z = M(r)
//                          p = z - beta p_prev,   beta  = (z, A p_prev) / (p_prev, A p_prev)
//                          x += alpha p,          alpha = (p, r) / (p, A p)
//                          r = b - A x            (the true residual, FP64)
//
// Two passes per iteration.  Pass 1 is one stencil pass over z giving
// (z, Az), (Az, p_prev) = (z, A p_prev) (A is symmetric), (z, r) and
// (p_prev, r); beta, (p, Ap) = (z,Az) - 2 beta (z,A p_prev) + beta^2 (p_prev,A p_prev)
// and alpha follow without forming q = A p.  Pass 2 writes p and x + alpha p
// and recomputes r = b - A x from them (neighbours formed on the fly), so the
// residual never drifts from the iterate and no final residual pass is needed.
// x and p alternate between two buffers by iteration parity (flags[1], on the
// device), so every iteration launches the same kernels on the same pointers
// and can be captured once in a graph.  x, b and the screening are FP64 and
// dense; z and r32 (the FP32 padded copy of r that the next V-cycle reads) are
// padded FP32; the direction p is stored in FP32 (dense): x moves along the
// unrounded z - beta p_prev, the stored copy only orthogonalises the next
// direction, and the residual is recomputed from x in FP64 every iteration,
// so the rounding perturbs alpha and beta by ~1e-7 relative and never the
// measured residual.
#include <type_traits>

#include "batch.cuh"
#include "common.cuh"
#include "occupancy.cuh"

namespace pb {
namespace fcg {

// Planes per block of the two passes unless the autotuner chose otherwise.  A block
// walks its planes one after another, so small grids take fewer planes for more
// blocks: at 65^3, 24 planes leave 81 blocks of pass 2 for 148 SMs (26.6 us), 4 planes
// 459; pass 1 at 257^3 takes 85 us with 24 planes and 79 with 12, at 513^3 419 and 443.
// (Times here and below are of a pass by itself, the L2 overwritten before it; inside a solve
// pass 1 takes 62 us at 257^3 and 386 at 513^3, pass 2 131 and 978.)
// Partial sums are sized for the shallowest depth a launch may use, kMinTZ.
constexpr int kTZ = 24, kMinTZ = 4, kThreads = 128;
__host__ __device__ constexpr int update_planes_of(int n) { return n <= 65 ? 4 : n <= 129 ? 8 : kTZ; }
__host__ __device__ constexpr int direction_planes_of(int n) { return n <= 65 ? 4 : n <= 129 ? 8 : n <= 257 ? 12 : kTZ; }

// Pass 2 tile: 32 x 8 nodes per block, kTZ planes deep.
constexpr int kUX = 32, kUY = 8, kUThreads = kUX * kUY;
static_assert(2 * (kUX + kUY) <= kUThreads, "one halo node per thread");

struct Pad {  // padded FP32 layout of the multigrid levels
    int n, P;
    int64_t plane;
    __device__ __forceinline__ int64_t at(int x, int y, int z) const {
        return checked_at(((int64_t)(z + 1) * (n + 2) + (y + 1)) * P + (x + 4), (int64_t)(n + 2) * plane, kSitePad);
    }
};

__device__ __forceinline__ int lin_tid() { return threadIdx.y * blockDim.x + threadIdx.x; }

// Sums K values over the block; results valid in linear thread 0.
template <int K>
__device__ __forceinline__ void block_sums(double (&v)[K], double (*shared)[32]) {
    const int tid = lin_tid(), lane = tid & 31, warp = tid >> 5;
    const int warps = (blockDim.x * blockDim.y) >> 5;
#pragma unroll
    for (int k = 0; k < K; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < K; ++k) shared[k][warp] = v[k];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = lane < warps ? shared[k][lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        }
    }
}

__device__ __forceinline__ int64_t block_index() {
    return ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
}

// The multiply-adds of both passes are written out: left to the compiler, two
// instantiations of a body (single and grouped launches, planes known or not) may
// fuse differently, and a cloud would differ in the last bits alone and in a batch.

constexpr int kW = 4;  // x per thread of pass 1
template <bool ALIGNED>  // the padded arrays start on 16-byte boundaries, and so do their rows
__device__ __forceinline__ float4 wide(const float* at) {
    if constexpr (ALIGNED) return *reinterpret_cast<const float4*>(at);
    return make_float4(at[0], at[1], at[2], at[3]);
}
static bool aligned16(const void* a, const void* b) { return ((uintptr_t)a | (uintptr_t)b) % 16 == 0; }
__device__ __forceinline__ void widen(float4 f, double (&d)[kW]) {
    d[0] = (double)f.x;
    d[1] = (double)f.y;
    d[2] = (double)f.z;
    d[3] = (double)f.w;
}

// (A v)_i: degree and screening at the node, its value and its neighbours' sum s.
__device__ __forceinline__ double applied(int degree, double pw, double screen, double h2, double value, double s) {
    return __fma_rn(__fma_rn(__dmul_rn(pw, screen), h2, __dmul_rn((double)degree, h2)), value, -__dmul_rn(s, h2));
}

// Pass 1: per-block (z, Az), (Az, p_prev), (z, r32), (p_prev, r32); flags[1]
// (iterations done) selects p_prev = p[it & 1]; flags[0] != 0 on the first step.
// A thread takes four x of a row (the padded rows start 16-byte aligned) and
// marches down z with the planes k - 1 and k in registers as doubles; the ghosts of
// the padded z are zero, so the 6-neighbour sum needs no tests, and the nodes past a
// row's end add zeros.  Bound by latency and by the conversions to double (16 a cycle
// and SM), not by memory: one x per thread converts 8 values a node and reads the
// screen everywhere (513^3: 508 us), four x 5.5 and the screen only where it is
// not zero (419; two x 495).
template <bool ALIGNED>
__device__ __forceinline__ void direction_sums_body(const float* __restrict__ z, Pad g, const float* __restrict__ p0,
                                                    const float* __restrict__ p1, const float* __restrict__ r32,
                                                    const double* __restrict__ screen,
                                                    const uint32_t* __restrict__ occupied, double pw,
                                                    const int* __restrict__ flags, double* __restrict__ part, int tz,
                                                    int bx, int by, int64_t block) {
    __shared__ double shared[4][32];
    const int n = g.n;
    const unsigned groups = (unsigned)(n + kW - 1) / kW;
    const unsigned t = bx * kThreads + threadIdx.x;  // flattened over the plane's (group, y): full warps
    const int y = (int)(t / groups), x = (int)(t - y * groups) * kW;
    const int z0 = by * tz, z1 = min(n, z0 + tz);
    const double h = (double)(n - 1), h2 = h * h;
    const bool first = flags[0] != 0;
    const float* __restrict__ pp = (flags[1] & 1) ? p1 : p0;
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    if (y < n) {
        const int degy = (y > 0) + (y + 1 < n);
        const int64_t nn = (int64_t)n * n;
        const int inside = min(kW, n - x);
        int64_t i = (int64_t)z0 * nn + (int64_t)y * n + x, c = g.at(x, y, z0);
        int some = (int)plane_bits(occupied, n, x, y, z0);  // signed: without a map the shifts leave it all ones
        double zb[kW], zm[kW];
        widen(wide<ALIGNED>(z + c - g.plane), zb);
        widen(wide<ALIGNED>(z + c), zm);
        for (int k = z0; k < z1; ++k, i += nn, c += g.plane, some >>= 1) {
            const float4 above = wide<ALIGNED>(z + c + g.plane);  // the ghost plane past the last
            const float4 front = wide<ALIGNED>(z + c - g.P), back = wide<ALIGNED>(z + c + g.P), res = wide<ALIGNED>(r32 + c);
            const float left = z[c - 1], right = z[c + kW];
            float prev[kW] = {};
            if (!first)
#pragma unroll
                for (int j = 0; j < kW; ++j)
                    if (j < inside) prev[j] = pp[i + j];
            double sc[kW] = {};
            if (some & 1)
#pragma unroll
                for (int j = 0; j < kW; ++j)
                    if (j < inside) sc[j] = screen[i + j];
            double za[kW], ym[kW], yp[kW], rc[kW];
            widen(above, za);
            widen(front, ym);
            widen(back, yp);
            widen(res, rc);
            const int degyz = degy + (k > 0) + (k + 1 < n);
#pragma unroll
            for (int j = 0; j < kW; ++j) {
                const double s = (j > 0 ? zm[j - 1] : (double)left) + (j < kW - 1 ? zm[j + 1] : (double)right) + ym[j] +
                                 yp[j] + zb[j] + za[j];
                const int deg = degyz + (j > 0 || x > 0) + (x + j + 1 < n);
                const double az = applied(deg, pw, sc[j], h2, zm[j], s), pv = (double)prev[j];
                v[0] = __fma_rn(zm[j], az, v[0]);
                v[1] = __fma_rn(az, pv, v[1]);
                v[2] = __fma_rn(zm[j], rc[j], v[2]);
                v[3] = __fma_rn(pv, rc[j], v[3]);
            }
#pragma unroll
            for (int j = 0; j < kW; ++j) {
                zb[j] = zm[j];
                zm[j] = za[j];
            }
        }
    }
    block_sums<4>(v, shared);
    if (lin_tid() == 0)
#pragma unroll
        for (int k = 0; k < 4; ++k) part[4 * block + k] = v[k];
}

// MINB: resident blocks per SM the compiler must allow (register budget); the
// autotuner picks among the compiled variants (PB_TUNE_FCG_DIRECTION_VARIANT).
template <int MINB, bool ALIGNED = true>
__global__ void __launch_bounds__(kThreads, MINB) direction_sums_kernel(const float* __restrict__ z, Pad g,
                                                                     const float* __restrict__ p0,
                                                                     const float* __restrict__ p1,
                                                                     const float* __restrict__ r32,
                                                                     const double* __restrict__ screen,
                                                                     const uint32_t* __restrict__ occupied, double pw,
                                                                     const int* __restrict__ flags,
                                                                     double* __restrict__ part, int tz) {
    direction_sums_body<ALIGNED>(z, g, p0, p1, r32, screen, occupied, pw, flags, part, tz, blockIdx.x, blockIdx.y, block_index());
}

// Sums pass 1's partials (fixed order) and forms the step's scalars:
//   scal[0] (p, Ap) (the previous direction's on entry)   scal[1] beta
//   scal[2] alpha   scal[3] (p, r)
__device__ __forceinline__ void direction_finish_body(const double* __restrict__ part, int blocks,
                                                      const int* __restrict__ flags, double* __restrict__ scal) {
    __shared__ double shared[4][32];
    double v[4] = {0.0, 0.0, 0.0, 0.0};
    for (int b = threadIdx.x; b < blocks; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] += part[4 * (int64_t)b + k];
    block_sums<4>(v, shared);
    if (threadIdx.x != 0) return;
    const double zz = v[0], zq = v[1], zr = v[2], pr = v[3];
    const bool first = flags[0] != 0;
    const double pap_prev = scal[0];
    const double beta = first || !(pap_prev > 0.0) ? 0.0 : zq / pap_prev;
    const double pap =
        first ? zz : __fma_rn(__dmul_rn(beta, beta), pap_prev, __fma_rn(__dmul_rn(-2.0, beta), zq, zz));
    const double prn = first ? zr : __fma_rn(-beta, pr, zr);
    scal[0] = pap;
    scal[1] = beta;
    scal[2] = pap > 0.0 ? prn / pap : 0.0;
    scal[3] = prn;
}

__global__ void direction_finish_kernel(const double* __restrict__ part, int blocks, const int* __restrict__ flags,
                                        double* __restrict__ scal) {
    direction_finish_body(part, blocks, flags, scal);
}

// Halo node of thread tid for a tile at (bx, by): rows by - 1 and by + kUY,
// columns bx - 1 and bx + kUX; (sx, sy) its slot in the shared tile.
struct Halo {
    int hx = -1, hy = -1, sx = 0, sy = 0;
    bool has = false;
    __device__ Halo(int tid, int bx, int by) {
        if (tid < 2 * kUX) {
            hx = bx + (tid % kUX);
            hy = tid < kUX ? by - 1 : by + kUY;
            sx = tid % kUX + 1;
            sy = tid < kUX ? 0 : kUY + 1;
            has = true;
        } else if (tid < 2 * kUX + 2 * kUY) {
            const int j = tid - 2 * kUX;
            hy = by + (j % kUY);
            hx = j < kUY ? bx - 1 : bx + kUX;
            sy = j % kUY + 1;
            sx = j < kUY ? 0 : kUX + 1;
            has = true;
        }
    }
    __device__ bool inside(int n) const { return has && hx >= 0 && hx < n && hy >= 0 && hy < n; }
};

// Pass 2: p_new = z - beta p_prev, x_new = x + alpha p_new, r = b - A x_new
// (neighbour values of x_new formed on the fly), r32 = (float) r, per-block
// ||r||^2.  Buffers by parity: p_prev = p[it & 1] -> p_new = p[(it+1) & 1],
// x = x[it & 1] -> x_new = x[(it+1) & 1].
//
// A 32 x 8 tile marches down z: the new iterate of plane k over the tile and
// its one-node halo goes to shared memory once (two tiles by plane parity, so
// one barrier per plane), the column's planes k - 1 and k + 1 stay in
// registers (about 7 global loads per node instead of 23 with every neighbour
// formed from memory).  Nodes outside the domain hold 0 and
// the neighbour sum adds x-, x+, y-, y+, z-, z+ in that order.
//
// Each thread copies the values it will read of plane k + RING - 1 (its x, z, p, b
// and screen, the last two where the occupancy words have any, and its halo node's x, z,
// p) into its own shared-memory slots with cp.async while it works on plane k, so
// RING - 1 planes of loads are in flight per thread without holding registers; a
// thread only reads its own slots, so cp.async.wait_group suffices (the tile of new
// iterates keeps its barrier).  The march is unrolled by the ring, so that slots are
// constants, and a plane's part of an address is the block's: 155 instructions per 32
// nodes instead of 225, and bound by the shared-memory pipe (72 %) and issue (64 %).
// 257^3 157 -> 147 us, 513^3 1240 -> 1011.  Tried: two rows per thread with the loads
// ahead in registers (200 us at 257^3, it waits on them in order), and whole rows
// copied 16 bytes at a time for all threads (165 us: fewer wavefronts, more
// instructions).  RING = 3 by default, 4 as a tuning variant.
constexpr int kRing = 3;

__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int TZC, int RING = kRing>
__device__ __forceinline__ void update_residual_prefetch_body(
    const float* __restrict__ z, Pad g, float* p0, float* p1, double* x0, double* x1, const double* __restrict__ b,
    const double* __restrict__ screen, const uint32_t* __restrict__ occupied, double pw,
    const double* __restrict__ scal, const int* __restrict__ flags, float* __restrict__ r32,
    double* __restrict__ part, int tz, int tile_x, int tile_y, int tile_z, int64_t block) {
    static_assert(RING >= 3 && RING <= 4, "two or three planes in flight");
    constexpr int kHalo = 2 * (kUX + kUY);     // the threads tid < kHalo own a halo node
    __shared__ double tiles[RING][kUY + 2][kUX + 2];
    __shared__ double shared[1][32];
    __shared__ double rd[RING][3][kUThreads];  // own x, b, screen
    __shared__ double hd[RING][kHalo];         // halo x
    __shared__ float rf[RING][2][kUThreads];   // own z, p
    __shared__ float hf[RING][2][kHalo];       // halo z, p
    const int n = g.n;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * kUX + tx;
    const int bx = tile_x * kUX, by = tile_y * kUY;
    const int x = bx + tx, y = by + ty;
    const int tzv = TZC > 0 ? TZC : tz;
    const int z0 = tile_z * tzv, z1 = min(n, z0 + tzv);
    const double h = (double)(n - 1), h2 = h * h;
    const int odd = flags[1] & 1;
    const bool first = flags[0] != 0;
    const float* __restrict__ pp = odd ? p1 : p0;
    float* __restrict__ pn = odd ? p0 : p1;
    const double* __restrict__ xc = odd ? x1 : x0;
    double* __restrict__ xn = odd ? x0 : x1;
    const double minus_beta = first ? 0.0 : -scal[1], alpha = scal[2];
    const int64_t nn = (int64_t)n * n;
    const Halo hl(tid, bx, by);
    const bool halo_in = hl.inside(n);
    const bool inside = x < n && y < n;
    // offsets within a plane, dense and padded; the plane's own part is the same for the block
    const uint32_t e = inside ? (uint32_t)y * n + x : 0u, q = inside ? (uint32_t)(y + 1) * g.P + x + 4 : 0u;
    const uint32_t he = halo_in ? (uint32_t)hl.hy * n + hl.hx : 0u;
    const uint32_t hq = halo_in ? (uint32_t)(hl.hy + 1) * g.P + hl.hx + 4 : 0u;
    // planes of the block where a warp's row of the tile has b or screening
    const uint32_t some =
        y < n ? plane_bits(occupied, n, bx, y, z0) & (0xffffffffu >> max(0, 32 - (z1 - z0))) : 0u;
    auto has_source = [&](int k) -> bool {  // deeper blocks than a word come without a map: every bit set
        return TZC > 0 && TZC <= 32 ? some >> (k - z0) & 1u : (int)some >> min(k - z0, 31) & 1;
    };
    // A slot that nothing is copied to holds zeros: nodes outside the domain, and p in the first step.
    for (int sl = 0; sl < RING; ++sl) {
        if (!inside) rd[sl][0][tid] = 0.0, rf[sl][0][tid] = 0.0f;
        if (!inside || first) rf[sl][1][tid] = 0.0f;
        if (hl.has) {
            if (!halo_in) hd[sl][tid] = 0.0, hf[sl][0][tid] = 0.0f;
            if (!halo_in || first) hf[sl][1][tid] = 0.0f;
        }
    }
    // plane k's values into its slot, one commit group; own x, z, p of planes z0 .. z1
    // (z1: the last plane's upper neighbour), the rest of z0 .. z1 - 1
    auto issue = [&](auto slot, int k) {
        constexpr int sl = decltype(slot)::value;
        const int64_t dense = k * nn, padded = (int64_t)(k + 1) * g.plane;
        if (inside && k <= z1 && k < n) {
            cp_async8(&rd[sl][0][tid], xc + dense + e);
            cp_async4(&rf[sl][0][tid], z + padded + q);
            if (!first) cp_async4(&rf[sl][1][tid], pp + dense + e);
            if (k < z1 && has_source(k)) {
                cp_async8(&rd[sl][1][tid], b + dense + e);
                cp_async8(&rd[sl][2][tid], screen + dense + e);
            }
        }
        if (halo_in && k < z1) {
            cp_async8(&hd[sl][tid], xc + dense + he);
            cp_async4(&hf[sl][0][tid], z + padded + hq);
            if (!first) cp_async4(&hf[sl][1][tid], pp + dense + he);
        }
        cp_commit();
    };
    issue(std::integral_constant<int, 0>(), z0);
    issue(std::integral_constant<int, 1>(), z0 + 1);
    if (RING == 4) issue(std::integral_constant<int, 2>(), z0 + 2);
    cp_wait<RING - 2>();
    double dm = __fma_rn(minus_beta, (double)rf[0][1][tid], (double)rf[0][0][tid]);
    double xm = __fma_rn(alpha, dm, rd[0][0][tid]), xb = 0.0;
    if (inside && z0 > 0) {
        const int64_t dense = (z0 - 1) * nn + e;
        double d = (double)z[(int64_t)z0 * g.plane + q];
        if (!first) d = __fma_rn(minus_beta, (double)pp[dense], d);
        xb = __fma_rn(alpha, d, xc[dense]);
    }
    // the diagonal without screening, between two planes and at the first or last
    const int degxy = (x > 0) + (x + 1 < n) + (y > 0) + (y + 1 < n);
    const double d_mid = __dmul_rn((double)(degxy + 2), h2), d_end = __dmul_rn((double)(degxy + 1), h2);
    double v[1] = {0.0};
    auto step = [&](auto slot, int k) {
        constexpr int sk = decltype(slot)::value, sn = (sk + 1) % RING;
        issue(std::integral_constant<int, (sk + RING - 1) % RING>(), k + RING - 1);  // plane k - 1's slot: its reader is this thread
        cp_wait<RING - 2>();  // planes up to k + 1 have landed
        double(*tile)[kUX + 2] = tiles[sk];
        tile[ty + 1][tx + 1] = xm;
        if (hl.has)
            tile[hl.sy][hl.sx] = __fma_rn(
                alpha, __fma_rn(minus_beta, (double)hf[sk][1][tid], (double)hf[sk][0][tid]), hd[sk][tid]);
        const bool up = k + 1 < n;
        const double da = __fma_rn(minus_beta, (double)rf[sn][1][tid], (double)rf[sn][0][tid]);
        const double xa = up ? __fma_rn(alpha, da, rd[sn][0][tid]) : 0.0;
        __syncthreads();
        if (inside) {
            const double s = tile[ty + 1][tx] + tile[ty + 1][tx + 2] + tile[ty][tx + 1] + tile[ty + 2][tx + 1] + xb + xa;
            double bi = 0.0, d = up && k > 0 ? d_mid : d_end;
            if (has_source(k)) {
                bi = rd[sk][1][tid];
                d = __fma_rn(__dmul_rn(pw, rd[sk][2][tid]), h2, d);
            }
            const double r = __dsub_rn(bi, __fma_rn(d, xm, -__dmul_rn(s, h2)));
            const int64_t dense = k * nn, padded = (int64_t)(k + 1) * g.plane;
            PB_GUARD(dense + e, nn * n, kSiteFcgStore) {
                pn[dense + e] = (float)dm;
                xn[dense + e] = xm;
            }
            PB_GUARD(padded + q, (int64_t)(n + 2) * g.plane, kSiteFcgStore)
            r32[padded + q] = (float)r;
            v[0] = __fma_rn(r, r, v[0]);
        }
        xb = xm;
        xm = xa;
        dm = da;
    };
    for (int k = z0; k < z1; k += RING) {  // slots by plane modulo RING, known at compile time
        step(std::integral_constant<int, 0>(), k);
        if (k + 1 < z1) step(std::integral_constant<int, 1>(), k + 1);
        if (k + 2 < z1) step(std::integral_constant<int, 2>(), k + 2);
        if constexpr (RING == 4)
            if (k + 3 < z1) step(std::integral_constant<int, 3>(), k + 3);
    }
    cp_wait<0>();
    block_sums<1>(v, shared);
    if (lin_tid() == 0) part[block] = v[0];
}

template <int TZC, int RING = kRing>
__global__ void __launch_bounds__(kUThreads) update_residual_prefetch_kernel(
    const float* __restrict__ z, Pad g, float* p0, float* p1, double* x0, double* x1, const double* __restrict__ b,
    const double* __restrict__ screen, const uint32_t* __restrict__ occupied, double pw,
    const double* __restrict__ scal, const int* __restrict__ flags, float* __restrict__ r32,
    double* __restrict__ part, int tz) {
    update_residual_prefetch_body<TZC, RING>(z, g, p0, p1, x0, x1, b, screen, occupied, pw, scal, flags, r32, part, tz,
                                             blockIdx.x, blockIdx.y, blockIdx.z, block_index());
}

// out[0] = sum over blocks of part[b] (fixed order).
__device__ __forceinline__ void sum_body(const double* __restrict__ part, int blocks, double* __restrict__ out) {
    __shared__ double shared[1][32];
    double v[1] = {0.0};
    for (int b = threadIdx.x; b < blocks; b += blockDim.x) v[0] += part[b];
    block_sums<1>(v, shared);
    if (threadIdx.x == 0) out[0] = v[0];
}

__global__ void sum_kernel(const double* __restrict__ part, int blocks, double* __restrict__ out) {
    sum_body(part, blocks, out);
}

// End of one iteration: record ||r||^2, count it, clear the first-step flag
// and, inside a graph, set the WHILE condition: continue while
// ||r||^2 > target2 and fewer than min(max_iter, ctrl[1]) iterations have run.
//   flags[0] first-step flag, flags[1] iterations; ctrl[0] = target2, ctrl[1] = cap.
__global__ void loop_kernel(cudaGraphConditionalHandle handle, int use_handle, const double* __restrict__ scal,
                            const double* __restrict__ ctrl, int* __restrict__ flags, int max_iter,
                            double* __restrict__ history) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const int it = flags[1] + 1;
    flags[1] = it;
    flags[0] = 0;
    const double r2 = scal[4];
    if (history && it <= max_iter) history[it - 1] = r2;
    const bool more = r2 > ctrl[0] && it < max_iter && (double)it < ctrl[1];
    if (use_handle) cudaGraphSetConditional(handle, more ? 1u : 0u);
}

static int direction_planes(int n) {
    const int64_t tz = tuned(PB_TUNE_FCG_DIRECTION_PLANES, n, direction_planes_of(n));
    return tz < kMinTZ ? kMinTZ : (int)tz;
}
static int update_planes(int n) {
    const int64_t tz = tuned(PB_TUNE_FCG_UPDATE_PLANES, n, update_planes_of(n));
    return tz < kMinTZ ? kMinTZ : (int)tz;
}
static dim3 flat_grid_of(int n, int tz) {
    return dim3((n * ((n + kW - 1) / kW) + kThreads - 1) / kThreads, (n + tz - 1) / tz);
}
static dim3 tile_grid_of(int n, int tz) {
    return dim3((n + kUX - 1) / kUX, (n + kUY - 1) / kUY, (n + tz - 1) / tz);
}
static unsigned count(dim3 g) { return g.x * g.y * g.z; }
static unsigned blocks_of(int n) {  // the most either pass can launch (kMinTZ planes per block)
    const unsigned a = count(flat_grid_of(n, kMinTZ)), t = count(tile_grid_of(n, kMinTZ));
    return a > t ? a : t;
}
__host__ __device__ inline Pad pad_of(int n) {
    const int P = ((n + 5) + 7) & ~7;
    return Pad{n, P, (int64_t)(n + 2) * P};
}

// ---- grouped launches over a batch of clouds (batch.cuh) --------------------------
// Per cloud c: flags + 4c (first step, iterations, active), scal + 8c, its own
// partial-sum area.  The point weight travels as the bits of a double in aux[0].

__device__ __forceinline__ double aux_double(int64_t bits) { return __longlong_as_double((long long)bits); }

// ptr[0] z, ptr[1] p0, ptr[2] p1, ptr[3] r32, ptr[4] screen, ptr[5] partials, ptr[6] occupancy (or null).
__global__ void __launch_bounds__(kThreads, 6) direction_sums_grouped_kernel(const batch::GridDesc* __restrict__ descs,
                                                                             int count, const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    auto run = [&](auto aligned) {
        direction_sums_body<decltype(aligned)::value>(
            (const float*)d.ptr[0], pad_of((int)d.n), (const float*)d.ptr[1], (const float*)d.ptr[2],
            (const float*)d.ptr[3], (const double*)d.ptr[4], screen_map(d.ptr[6]), aux_double(d.aux[0]),
            flags + d.cloud * batch::kFlagStride, (double*)d.ptr[5], (int)d.aux[1], bx, by, bx + d.gx * (int64_t)by);
    };
    if (d.aux[2]) run(std::true_type());
    else run(std::false_type());
}

// One block per cloud: ptr[0] partials, ptr[1] the cloud's scalars; aux[0] pass-1 blocks.
__global__ void direction_finish_grouped_kernel(const batch::GridDesc* __restrict__ descs, int count,
                                                const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    direction_finish_body((const double*)d.ptr[0], (int)d.aux[0], flags + d.cloud * batch::kFlagStride,
                          (double*)d.ptr[1]);
}

// ptr[0] z, ptr[1] p0, ptr[2] p1, ptr[3] x0, ptr[4] x1, ptr[5] b, ptr[6] screen, ptr[7] r32, ptr[8] the
// cloud's scalars, ptr[9] partials, ptr[10] occupancy (or null).
__global__ void __launch_bounds__(kUThreads, 4) update_residual_grouped_kernel(const batch::GridDesc* __restrict__ descs,
                                                                            int count, const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    update_residual_prefetch_body<0>(
        (const float*)d.ptr[0], pad_of((int)d.n), (float*)d.ptr[1], (float*)d.ptr[2], (double*)d.ptr[3],
        (double*)d.ptr[4], (const double*)d.ptr[5], (const double*)d.ptr[6], either_map(d.ptr[10], (int)d.n),
        aux_double(d.aux[0]), (const double*)d.ptr[8], flags + d.cloud * batch::kFlagStride, (float*)d.ptr[7],
        (double*)d.ptr[9], (int)d.aux[1], bx, by, bz, bx + d.gx * ((int64_t)by + d.gy * bz));
}

// One block per cloud: ptr[0] partials, ptr[1] output (the cloud's scal + 4); aux[0] blocks.
__global__ void sum_grouped_kernel(const batch::GridDesc* __restrict__ descs, int count,
                                   const int* __restrict__ flags) {
    int bx, by, bz;
    const batch::GridDesc& d = batch::locate(descs, count, blockIdx.x, bx, by, bz);
    if (!batch::cloud_active(flags, d.cloud)) return;
    sum_body((const double*)d.ptr[0], (int)d.aux[0], (double*)d.ptr[1]);
}

// End of one batch iteration, every active cloud: record ||r||^2, count the
// iteration, clear the first-step flag, and keep the cloud active while
// ||r||^2 > target2 and fewer than min(max_iter, cap) iterations have run.  The
// WHILE condition (inside a graph) continues while any cloud is active.
__global__ void __launch_bounds__(1024) loop_batch_kernel(cudaGraphConditionalHandle handle, int use_handle,
                                                          const double* __restrict__ scal,
                                                          const double* __restrict__ ctrl, int* __restrict__ flags,
                                                          int clouds, int max_iter, double* __restrict__ history) {
    int any = 0;
    for (int c = threadIdx.x; c < clouds; c += blockDim.x) {
        int* f = flags + (int64_t)c * batch::kFlagStride;
        if (!f[batch::kFlagActive]) continue;
        const int it = f[batch::kFlagIter] + 1;
        f[batch::kFlagIter] = it;
        f[batch::kFlagFirst] = 0;
        const double r2 = scal[(int64_t)c * batch::kScalStride + 4];
        if (history && it <= max_iter) history[(int64_t)c * max_iter + it - 1] = r2;
        const double* ct = ctrl + (int64_t)c * batch::kCtrlStride;
        const bool more = r2 > ct[0] && it < max_iter && (double)it < ct[1];
        f[batch::kFlagActive] = more ? 1 : 0;
        any |= more ? 1 : 0;
    }
    any = __syncthreads_or(any);
    if (use_handle && threadIdx.x == 0) cudaGraphSetConditional(handle, any ? 1u : 0u);
}

}  // namespace fcg

namespace batch {

int describe_fcg_direction(GridDesc& d) {
    const int n = (int)d.n;
    for (int k = 0; k < 6; ++k)
        if (!d.ptr[k]) return fail(PB_ERR_INVALID, "batch fcg direction: bad args");
    if (n < 2 || n > 4097 || d.ptr[1] == d.ptr[2]) return fail(PB_ERR_INVALID, "batch fcg direction: bad args");
    const int tz = fcg::direction_planes_of(n);  // grouped launches keep the built-in planes per block
    const dim3 g = fcg::flat_grid_of(n, tz);
    d.gx = g.x;
    d.gy = g.y;
    d.gz = 1;
    d.aux[1] = tz;
    d.aux[2] = fcg::aligned16(d.ptr[0], d.ptr[3]);
    return PB_OK;
}

int describe_fcg_update(GridDesc& d) {
    const int n = (int)d.n;
    for (int k = 0; k < 10; ++k)
        if (!d.ptr[k]) return fail(PB_ERR_INVALID, "batch fcg update: bad args");
    if (n < 2 || n > 4097 || d.ptr[1] == d.ptr[2] || d.ptr[3] == d.ptr[4])
        return fail(PB_ERR_INVALID, "batch fcg update: bad args");
    const int tz = fcg::update_planes_of(n);
    const dim3 g = fcg::tile_grid_of(n, tz);
    d.gx = g.x;
    d.gy = g.y;
    d.gz = g.z;
    d.aux[1] = tz;
    return PB_OK;
}

int describe_fcg_reduce(GridDesc& d) {
    if (!d.ptr[0] || !d.ptr[1] || d.aux[0] < 1) return fail(PB_ERR_INVALID, "batch fcg reduce: bad args");
    d.gx = d.gy = d.gz = 1;
    return PB_OK;
}

// Partial-sum doubles one cloud of side n needs (both FCG passes).
int64_t fcg_partials(int n) { return (int64_t)fcg::blocks_of(n) * 4; }
int64_t fcg_direction_blocks(int n) { return fcg::count(fcg::flat_grid_of(n, fcg::direction_planes_of(n))); }
int64_t fcg_update_blocks(int n) { return fcg::count(fcg::tile_grid_of(n, fcg::update_planes_of(n))); }

int launch_fcg(int kind, const GridDesc* descs, int count, int64_t blocks, const int* flags, cudaStream_t s) {
    switch (kind) {
        case 0:
            fcg::direction_sums_grouped_kernel<<<(unsigned)blocks, fcg::kThreads, 0, s>>>(descs, count, flags);
            PB_CHECK_LAUNCH("direction_sums_grouped_kernel");
            return PB_OK;
        case 1:
            fcg::direction_finish_grouped_kernel<<<(unsigned)blocks, 1024, 0, s>>>(descs, count, flags);
            PB_CHECK_LAUNCH("direction_finish_grouped_kernel");
            return PB_OK;
        case 2:
            fcg::update_residual_grouped_kernel<<<(unsigned)blocks, dim3(fcg::kUX, fcg::kUY), 0, s>>>(descs, count,
                                                                                                      flags);
            PB_CHECK_LAUNCH("update_residual_grouped_kernel");
            return PB_OK;
        case 3:
            fcg::sum_grouped_kernel<<<(unsigned)blocks, 1024, 0, s>>>(descs, count, flags);
            PB_CHECK_LAUNCH("sum_grouped_kernel");
            return PB_OK;
    }
    return fail(PB_ERR_INVALID, "batch fcg: unknown kind %d", kind);
}

int launch_loop_batch(unsigned long long handle, const double* scal, const double* ctrl, int* flags, int clouds,
                      int max_iter, double* history, cudaStream_t s) {
    fcg::loop_batch_kernel<<<1, 1024, 0, s>>>((cudaGraphConditionalHandle)handle, handle != 0, scal, ctrl, flags,
                                              clouds, max_iter, history);
    PB_CHECK_LAUNCH("loop_batch_kernel");
    return PB_OK;
}

}  // namespace batch
}  // namespace pb

using namespace pb;

extern "C" size_t pb_fcg_workspace_size(int64_t n) {
    if (n < 2) n = 2;
    return (size_t)fcg::blocks_of((int)n) * 4 * sizeof(double) + 256;
}

static int fcg_check(int64_t n, size_t workspace_bytes, const void* workspace) {
    if (!workspace || workspace_bytes < (size_t)pb::fcg::blocks_of((int)n) * 4 * sizeof(double))
        return fail(PB_ERR_WORKSPACE, "fcg: workspace needs %zu bytes", pb_fcg_workspace_size(n));
    return PB_OK;
}

// FCG(1) pass 1 after the preconditioner produced z (padded FP32): the step's
// scalars into scal[0..3] (scal[0] holds the previous (p, Ap) on entry).
// p0/p1: the two dense FP32 direction buffers, p_prev = p[flags[1] & 1];
// r32: the padded FP32 residual the preconditioner read; occupancy: the words that
// pb_refine_start_f64 wrote for this screen and right-hand side, or null.
extern "C" int pb_fcg_direction_sparse_f64(const float* z, const float* p0, const float* p1, const float* r32,
                                           const double* screen, const void* occupancy, int64_t n,
                                           double point_weight, double* scal, const int* flags, void* workspace,
                                           size_t workspace_bytes, void* stream) {
    using namespace pb::fcg;
    if (n < 2 || n > 4097 || !z || !p0 || !p1 || p0 == p1 || !r32 || !screen || !scal || !flags)
        return fail(PB_ERR_INVALID, "fcg direction: bad args");
    PB_TRY(fcg_check(n, workspace_bytes, workspace));
    double* part = (double*)workspace;
    cudaStream_t s = (cudaStream_t)stream;
    const int tz = direction_planes((int)n);
    const dim3 grid = flat_grid_of((int)n, tz);
    auto dir = direction_sums_kernel<6>;
    switch (tuned(PB_TUNE_FCG_DIRECTION_VARIANT, n, 0)) {
        case 1: dir = direction_sums_kernel<4>; break;
        case 2: dir = direction_sums_kernel<8>; break;
        default: break;
    }
    if (!aligned16(z, r32)) dir = direction_sums_kernel<4, false>;
    dir<<<grid, kThreads, 0, s>>>(z, pad_of((int)n), p0, p1, r32, screen, tz <= 32 ? screen_map(occupancy) : nullptr,
                                  point_weight, flags, part, tz);
    PB_CHECK_LAUNCH("fcg direction_sums_kernel");
    direction_finish_kernel<<<1, 1024, 0, s>>>(part, (int)count(grid), flags, scal);
    PB_CHECK_LAUNCH("fcg direction_finish_kernel");
    return PB_OK;
}

extern "C" int pb_fcg_direction_f64(const float* z, const float* p0, const float* p1, const float* r32,
                                    const double* screen, int64_t n, double point_weight, double* scal,
                                    const int* flags, void* workspace, size_t workspace_bytes, void* stream) {
    return pb_fcg_direction_sparse_f64(z, p0, p1, r32, screen, nullptr, n, point_weight, scal, flags, workspace,
                                       workspace_bytes, stream);
}

// FCG(1) pass 2: p_new, x_new = x + alpha p_new and the true residual
// r = b - A x_new into r32, scal[4] = ||r||^2.  Iterate and direction buffers
// alternate by parity of flags[1]: x[it & 1] -> x[(it+1) & 1].  occupancy as in pass 1.
extern "C" int pb_fcg_update_sparse_f64(const float* z, float* p0, float* p1, double* x0, double* x1, const double* b,
                                        const double* screen, const void* occupancy, float* r32, int64_t n,
                                        double point_weight, double* scal, const int* flags, void* workspace,
                                        size_t workspace_bytes, void* stream) {
    using namespace pb::fcg;
    if (n < 2 || n > 4097 || !z || !p0 || !p1 || p0 == p1 || !x0 || !x1 || x0 == x1 || !b || !screen || !r32 ||
        !scal || !flags)
        return fail(PB_ERR_INVALID, "fcg update: bad args");
    PB_TRY(fcg_check(n, workspace_bytes, workspace));
    double* part = (double*)workspace;
    cudaStream_t s = (cudaStream_t)stream;
    const int tz = update_planes((int)n);
    const dim3 grid = tile_grid_of((int)n, tz);
    const bool fixed = tz == kTZ;
    auto upd = fixed ? update_residual_prefetch_kernel<kTZ> : update_residual_prefetch_kernel<0>;
    if (tuned(PB_TUNE_FCG_UPDATE_VARIANT, n, 0) == 4)
        upd = fixed ? update_residual_prefetch_kernel<kTZ, 4> : update_residual_prefetch_kernel<0, 4>;
    upd<<<grid, dim3(kUX, kUY), 0, s>>>(z, pad_of((int)n), p0, p1, x0, x1, b, screen,
                                        tz <= 32 ? either_map(occupancy, (int)n) : nullptr, point_weight, scal, flags,
                                        r32, part, tz);
    PB_CHECK_LAUNCH("fcg update_residual_prefetch_kernel");
    sum_kernel<<<1, 1024, 0, s>>>(part, (int)count(grid), scal + 4);
    PB_CHECK_LAUNCH("fcg sum_kernel");
    return PB_OK;
}

extern "C" int pb_fcg_update_f64(const float* z, float* p0, float* p1, double* x0, double* x1, const double* b,
                                 const double* screen, float* r32, int64_t n, double point_weight, double* scal,
                                 const int* flags, void* workspace, size_t workspace_bytes, void* stream) {
    return pb_fcg_update_sparse_f64(z, p0, p1, x0, x1, b, screen, nullptr, r32, n, point_weight, scal, flags, workspace,
                                    workspace_bytes, stream);
}

// ---- device-driven iteration: a CUDA graph with a WHILE conditional node ------
// pb_loop_capture_begin creates a graph holding one WHILE node and starts
// capturing `stream` into its body; the caller then queues one iteration (its
// last launch being pb_loop_condition with the returned handle) and calls
// pb_loop_capture_end, which instantiates the graph.  Each pb_graph_launch then
// runs iterations on the device until the condition kernel says stop — no
// host synchronisation per iteration.  The condition starts at 1 on every launch.
extern "C" int pb_loop_capture_begin(void* stream, void** graph_out, unsigned long long* handle_out) {
    if (!graph_out || !handle_out) return fail(PB_ERR_INVALID, "loop capture: null output");
    cudaGraph_t graph = nullptr;
    PB_CHECK_CUDA(cudaGraphCreate(&graph, 0), "cudaGraphCreate");
    cudaGraphConditionalHandle handle;
    cudaError_t e = cudaGraphConditionalHandleCreate(&handle, graph, 1, cudaGraphCondAssignDefault);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return cuda_fail(e, "cudaGraphConditionalHandleCreate");
    }
    cudaGraphNodeParams params = {};
    params.type = cudaGraphNodeTypeConditional;
    params.conditional.handle = handle;
    params.conditional.type = cudaGraphCondTypeWhile;
    params.conditional.size = 1;
    cudaGraphNode_t node;
    e = cudaGraphAddNode(&node, graph, nullptr, 0, &params);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return cuda_fail(e, "cudaGraphAddNode (while)");
    }
    cudaGraph_t body = params.conditional.phGraph_out[0];
    e = cudaStreamBeginCaptureToGraph((cudaStream_t)stream, body, nullptr, nullptr, 0,
                                      cudaStreamCaptureModeRelaxed);
    if (e != cudaSuccess) {
        cudaGraphDestroy(graph);
        return cuda_fail(e, "cudaStreamBeginCaptureToGraph");
    }
    *graph_out = graph;
    *handle_out = (unsigned long long)handle;
    return PB_OK;
}

// Queues the end-of-iteration kernel (see loop_kernel).  handle = 0: eager use
// outside a graph (no condition is set).
extern "C" int pb_loop_condition(unsigned long long handle, const double* scal, const double* ctrl, int* flags,
                                 int64_t max_iter, double* history, void* stream) {
    if (!scal || !ctrl || !flags || max_iter < 1) return fail(PB_ERR_INVALID, "loop condition: bad args");
    pb::fcg::loop_kernel<<<1, 32, 0, (cudaStream_t)stream>>>((cudaGraphConditionalHandle)handle, handle != 0, scal,
                                                            ctrl, flags, (int)max_iter, history);
    PB_CHECK_LAUNCH("loop_kernel");
    return PB_OK;
}

extern "C" int pb_loop_capture_end(void* stream, void* graph, void** exec_out) {
    if (!graph || !exec_out) return fail(PB_ERR_INVALID, "loop capture end: bad args");
    cudaGraph_t captured = nullptr;
    cudaError_t e = cudaStreamEndCapture((cudaStream_t)stream, &captured);
    if (e != cudaSuccess) {
        cudaGraphDestroy((cudaGraph_t)graph);
        return cuda_fail(e, "cudaStreamEndCapture");
    }
    cudaGraphExec_t exec = nullptr;
    e = cudaGraphInstantiate(&exec, (cudaGraph_t)graph, 0);
    if (e != cudaSuccess) {
        cudaGraphDestroy((cudaGraph_t)graph);
        return cuda_fail(e, "cudaGraphInstantiate");
    }
    *exec_out = exec;
    return PB_OK;
}

extern "C" int pb_graph_launch(void* exec, void* stream) {
    if (!exec) return fail(PB_ERR_INVALID, "graph launch: null graph");
    PB_CHECK_CUDA(cudaGraphLaunch((cudaGraphExec_t)exec, (cudaStream_t)stream), "cudaGraphLaunch");
    return PB_OK;
}

extern "C" int pb_graph_destroy(void* exec, void* graph) {
    if (exec) cudaGraphExecDestroy((cudaGraphExec_t)exec);
    if (graph) cudaGraphDestroy((cudaGraph_t)graph);
    return PB_OK;
}

// Adds launches that ran inside graphs (known to the host only afterwards) to
// the library's launch count.
extern "C" int pb_note_launches(long long count);
