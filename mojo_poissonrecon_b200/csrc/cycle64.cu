// One whole FP64 V-cycle of the reference per call (core.py:141-193), bit-exact.
//
// Every node update here computes what stencil64.cu's kernels compute, in the
// same order (-fmad=false): s = ((((x- + x+) + y-) + y+) + z-) + z+ with absent
// neighbours adding +0.0 (a sum that starts from +0.0 never becomes -0.0, so
// adding +0.0 changes no bit), then (rhs + s h^-2) / diagonal.
#include <map>
#include <mutex>

#include "common.cuh"

namespace pb {
namespace cycle64 {

// a / d for d = a level's diagonal, y = RN(1 / d): the quotient estimate a y is
// corrected twice with exact remainders (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", 1990).  After
// the first correction the quotient is within one ulp of a / d, and by
// Markstein's theorem the second then rounds correctly, for any a and d whose
// products and remainders neither overflow nor underflow; divide() tests the
// exponents for that and takes the general division elsewhere.
// Five dependent multiply-adds against the general division's longer chain.
__device__ __forceinline__ double divide(double a, double d, double y) {
    const uint32_t e = (uint32_t)__double2hiint(a) & 0x7ff00000u;
    if (y != 0.0 && e - (123u << 20) <= (1800u << 20)) {  // |a| in [2^-900, 2^901)
        double q = a * y;
        q = __fma_rn(__fma_rn(-d, q, a), y, q);
        return __fma_rn(__fma_rn(-d, q, a), y, q);
    }
    return a == 0.0 && d > 0.0 ? a : a / d;
}

// RN(1 / d) where divide() may use it (|d| in [2^-99, 2^100], a positive diagonal), else 0.
__device__ __forceinline__ double reciprocal(double d) {
    return d >= 0x1p-99 && d <= 0x1p100 ? 1.0 / d : 0.0;
}

// ---- the coarse tail: levels of side <= 17 in one block ---------------------------
//
// What bounded the per-level launches: a V-cycle makes 80 one-colour passes on
// the 3^3 grid and 17 launches on each of 5^3, 9^3 and 17^3, 2-3 us apiece
// whatever they compute.  Here one block keeps every level's iterate, right-hand
// side, diagonal and reciprocal in shared memory (225 KB from 17^3 down) and a
// phase costs a barrier and a shared-memory round trip.  Levels of side 9, 5
// and 3 run on the first 384, 64 and 32 threads (their nodes of one colour)
// with named barriers of that many threads.  Measured on B200: a depth-5
// reconstruction of 2,000 points (five cycles) 3.56 -> 1.21 ms, 13,337 points
// at depth 6 (four cycles) 3.38 -> 1.48 ms; 0.9 and 1.2 ms since 33^3 and 17^3 run
// in a cluster (below), which leaves this kernel the devices that cannot place one.
//
// A side is odd, so the colour of a node is the lowest bit of its linear index i
// and its six neighbours (i +- 1, i +- N, i +- N^2) have the other colour: each
// array holds colour 0 then colour 1, node i at i / 2 of its colour, which makes a
// warp's accesses contiguous (dense, every access was four wavefronts instead of
// two, and a one-colour pass over 17^3 is bound by them).
constexpr int kTailThreads = 672;  // 80 registers a thread; a colour of 17^3 in four rounds

template <int N>
struct Tail {
    static constexpr int kNodes = N * N * N, kHalf = (kNodes + 1) / 2;
    static constexpr int kThreads = N >= 17 ? kTailThreads : N == 9 ? 384 : N == 5 ? 64 : 32;
    double sol[2][kHalf + 1];  // the last entry of each colour stays +0.0: an absent neighbour
    double rhs[2][kHalf];
    double diag[2][kHalf];
    double inv[2][kHalf];
};

template <int N>
__device__ __forceinline__ void tail_barrier() {
    if (N == 3) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"n"(N >= 17 ? 1 : N == 9 ? 2 : 3), "n"(Tail<N>::kThreads) : "memory");
}

// The six neighbours' entries of node i, absent ones at the zero entry.
template <int N>
struct Around {
    int at[6];
    __device__ __forceinline__ explicit Around(int i) {
        const int x = i % N, row = i / N, y = row % N, z = row / N, none = Tail<N>::kHalf;
        at[0] = x > 0 ? (i - 1) >> 1 : none;
        at[1] = x + 1 < N ? (i + 1) >> 1 : none;
        at[2] = y > 0 ? (i - N) >> 1 : none;
        at[3] = y + 1 < N ? (i + N) >> 1 : none;
        at[4] = z > 0 ? (i - N * N) >> 1 : none;
        at[5] = z + 1 < N ? (i + N * N) >> 1 : none;
    }
    // v: the other colour.  The reference's sum starts from +0.0, so it is +0.0 where six -0.0 meet: the right-hand
    // sides here are never -0.0 (restricted sums start from +0.0, the finest one is read as 0.0 + rhs), and
    // rhs + s h^-2 is then the same for either zero.
    __device__ __forceinline__ double sum(const double* v) const {
        return ((((v[at[0]] + v[at[1]]) + v[at[2]]) + v[at[3]]) + v[at[4]]) + v[at[5]];
    }
};

template <int N>
__device__ __forceinline__ void tail_update(Tail<N>& L, int colour, int p, const Around<N>& a) {
    const double h2 = (double)(N - 1) * (double)(N - 1);
    const double s = a.sum(L.sol[1 - colour]), d = L.diag[colour][p];
    if (d > 1.0e-30) L.sol[colour][p] = divide(__fma_rn(s, h2, L.rhs[colour][p]), d, L.inv[colour][p]);  // s h2 is exact
}

// Sweeps of level N; every thread below kThreads takes part.
template <int N>
__device__ __forceinline__ void tail_relax(Tail<N>& L, int sweeps) {
    const int tid = threadIdx.x;
    if constexpr (N <= 9) {  // at most one node of each colour per thread: addresses once
        const bool in0 = 2 * tid < Tail<N>::kNodes, in1 = 2 * tid + 1 < Tail<N>::kNodes;
        const Around<N> a(in0 ? 2 * tid : 0), b(in1 ? 2 * tid + 1 : 1);
        for (int it = 0; it < sweeps; ++it) {
            if (in0) tail_update<N>(L, 0, tid, a);
            tail_barrier<N>();
            if (in1) tail_update<N>(L, 1, tid, b);
            tail_barrier<N>();
        }
    } else {
        for (int phase = 0; phase < 2 * sweeps; ++phase) {
            const int colour = phase & 1;
#pragma unroll 1  // registers: unrolled, every round's addresses are kept and spilled
            for (int p = tid; 2 * p + colour < Tail<N>::kNodes; p += Tail<N>::kThreads)
                tail_update<N>(L, colour, p, Around<N>(2 * p + colour));
            tail_barrier<N>();
        }
    }
}

template <int N>
__device__ __forceinline__ void tail_residual(const Tail<N>& L, double* __restrict__ res) {
    const double h2 = (double)(N - 1) * (double)(N - 1);
#pragma unroll 1
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += Tail<N>::kThreads) {
        const int c = i & 1, p = i >> 1;
        const double s = Around<N>(i).sum(L.sol[1 - c]);
        res[i] = L.rhs[c][p] - (L.diag[c][p] * L.sol[c][p] - s * h2);
    }
}

// capi.mojo:557-673 from the fine residual; the coarse iterate starts at zero.
template <int N, int C>
__device__ __forceinline__ void tail_restrict(const double* __restrict__ res, Tail<C>& L) {
#pragma unroll 1
    for (int i = threadIdx.x; i < Tail<C>::kNodes; i += Tail<N>::kThreads) {
        const int x = i % C, y = (i / C) % C, z = i / (C * C);
        double sum = 0.0, weight = 0.0;
#pragma unroll 1  // registers
        for (int oz = -1; oz <= 1; ++oz)
#pragma unroll
            for (int oy = -1; oy <= 1; ++oy)
#pragma unroll
                for (int ox = -1; ox <= 1; ++ox) {
                    const int zz = 2 * z + oz, yy = 2 * y + oy, xx = 2 * x + ox;
                    const double w = (oz ? 1.0 : 2.0) * (oy ? 1.0 : 2.0) * (ox ? 1.0 : 2.0);
                    if ((unsigned)zz < N && (unsigned)yy < N && (unsigned)xx < N) {
                        sum += res[(zz * N + yy) * N + xx] * w;
                        weight += w;
                    }
                }
        L.rhs[i & 1][i >> 1] = sum / weight;
        L.sol[i & 1][i >> 1] = 0.0;
    }
}

// capi.mojo:677-742
template <int N, int C>
__device__ __forceinline__ void tail_prolong(Tail<N>& L, const Tail<C>& K) {
#pragma unroll 1
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += Tail<N>::kThreads) {
        const int x = i % N, y = (i / N) % N, z = i / (N * N);
        const int x0 = x / 2, y0 = y / 2, z0 = z / 2;
        const int x1 = min(x0 + 1, C - 1), y1 = min(y0 + 1, C - 1), z1 = min(z0 + 1, C - 1);
        const double tx = (x & 1) ? 0.5 : 0.0, ty = (y & 1) ? 0.5 : 0.0, tz = (z & 1) ? 0.5 : 0.0;
        auto at = [&](int xx, int yy, int zz) {
            const int j = (zz * C + yy) * C + xx;
            return K.sol[j & 1][j >> 1];
        };
        const double c00 = at(x0, y0, z0) * (1.0 - tx) + at(x1, y0, z0) * tx;
        const double c10 = at(x0, y1, z0) * (1.0 - tx) + at(x1, y1, z0) * tx;
        const double c01 = at(x0, y0, z1) * (1.0 - tx) + at(x1, y0, z1) * tx;
        const double c11 = at(x0, y1, z1) * (1.0 - tx) + at(x1, y1, z1) * tx;
        const double c0 = c00 * (1.0 - ty) + c10 * ty;
        const double c1 = c01 * (1.0 - ty) + c11 * ty;
        L.sol[i & 1][i >> 1] += c0 * (1.0 - tz) + c1 * tz;
    }
}

template <int N>
struct TailStack {
    Tail<N> level;
    TailStack<(N + 1) / 2> below;
};
template <>
struct TailStack<3> {
    Tail<3> level;
};

template <int N>
struct TailSmem {
    double residual[N * N * N];  // of whichever level is being restricted
    TailStack<N> stack;
};

// Diagonals and reciprocals of every level from the screens, and the zero entries.
template <int N>
__device__ __forceinline__ void tail_setup(TailStack<N>& S, const double* const* screens, double pw) {
    const double h2 = (double)(N - 1) * (double)(N - 1);
    const double* __restrict__ screen = screens[0];
#pragma unroll 2
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += kTailThreads) {
        const int x = i % N, y = (i / N) % N, z = i / (N * N);
        const int degree = (x > 0) + (x + 1 < N) + (y > 0) + (y + 1 < N) + (z > 0) + (z + 1 < N);
        const double d = (double)degree * h2 + pw * screen[i] * h2;
        S.level.diag[i & 1][i >> 1] = d;
        S.level.inv[i & 1][i >> 1] = reciprocal(d);
    }
    if (threadIdx.x < 2) S.level.sol[threadIdx.x][Tail<N>::kHalf] = 0.0;
    if constexpr (N > 3) tail_setup<(N + 1) / 2>(S.below, screens + 1, pw);
}

template <int N>
__device__ __forceinline__ void tail_cycle(TailStack<N>& S, double* res, int pre, int post) {
    if constexpr (N == 3) {
        tail_relax<3>(S.level, 40);
    } else {
        constexpr int C = (N + 1) / 2;
        tail_relax<N>(S.level, pre);
        tail_residual<N>(S.level, res);
        tail_barrier<N>();
        tail_restrict<N, C>(res, S.below.level);
        tail_barrier<N>();
        if (threadIdx.x < Tail<C>::kThreads) tail_cycle<C>(S.below, res, pre, post);
        tail_barrier<N>();
        tail_prolong<N, C>(S.level, S.below.level);
        tail_barrier<N>();
        tail_relax<N>(S.level, post);
    }
}

struct TailArgs {
    const double* screens[5];  // top level first
    const double* rhs;         // of the top level
    double* sol;               // of the top level: the iterate, or (zero_start) written only
    double pw;
    int pre, post, cycles, zero_start;
};

template <int N>
__global__ void __launch_bounds__(kTailThreads) tail_kernel(const TailArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    TailSmem<N>& S = *reinterpret_cast<TailSmem<N>*>(raw);
    tail_setup<N>(S.stack, a.screens, a.pw);
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += kTailThreads) {
        S.stack.level.rhs[i & 1][i >> 1] = 0.0 + a.rhs[i];
        S.stack.level.sol[i & 1][i >> 1] = a.zero_start ? 0.0 : a.sol[i];
    }
    __syncthreads();
    for (int c = 0; c < a.cycles; ++c) {
        if (threadIdx.x < Tail<N>::kThreads) tail_cycle<N>(S.stack, S.residual, a.pre, a.post);
        __syncthreads();
    }
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += kTailThreads) a.sol[i] = S.stack.level.sol[i & 1][i >> 1];
}

// ---- levels 33 and 17 over a cluster of 16 blocks ---------------------------------
//
// 33^3 does not fit one block, and as grid launches its twelve one-colour passes,
// restriction and prolongation take 41 us a cycle, nearly all of it launch latency;
// 17^3 in one block is bound by that SM's shared-memory accesses (19 us).  Here a
// cluster of 16 blocks keeps both levels in distributed shared memory as z slabs
// (two planes of 33^3 and one of 17^3 each, the last block one more), a block holds
// a copy of the plane on either side of its slab, and an update of a slab's first or
// last plane is stored to the neighbour's copy too; a phase then ends with one
// cluster barrier.  The levels below run on block 0 as above.  A node's index,
// colour and place follow the rule of the tail with the block's own even origin.
// Measured on B200: a V(3,3) cycle from 33^3 down 124 -> 68 us within a call of several
// (336 us for the five of a depth-5 reconstruction); a call of one takes 95, set-up included.
constexpr int kClusterBlocks = 16, kClusterThreads = 832;  // 1634 nodes of a colour (last block) in two rounds

template <int N, int PLANES>
struct Slab {
    static constexpr int kNN = N * N, kSol = ((PLANES + 2) * kNN + 3) / 2, kOwn = (PLANES * kNN + 3) / 2;
    double sol[2][kSol + 1];  // the last entry stays +0.0: an absent x or y neighbour; absent planes stay +0.0 too
    double rhs[2][kOwn];
    double diag[2][kOwn];
    double inv[2][kOwn];
};

// The planes [first, last) of block `rank`, and the even origin of its node indices (below plane first - 1).
template <int N>
struct SlabPlace {
    static constexpr int kNN = N * N, kStep = (N - 1) / kClusterBlocks;
    int first, last, origin, own;  // own: packed index of the slab's first pair of nodes
    __device__ __forceinline__ explicit SlabPlace(int rank)
        : first(kStep * rank), last(rank + 1 < kClusterBlocks ? first + kStep : N),
          origin(((first - 1) * kNN) & ~1), own((first * kNN - origin) >> 1) {}
};

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// The address in block `rank` of this block's shared variable.
__device__ __forceinline__ uint32_t remote_address(const void* local, uint32_t rank) {
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"((uint32_t)__cvta_generic_to_shared(local)), "r"(rank));
    return out;
}
__device__ __forceinline__ void remote_store(uint32_t address, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(address), "d"(v) : "memory");
}
__device__ __forceinline__ double remote_load(uint32_t address) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(address) : "memory");
    return v;
}

// Stores node i's value to the neighbour's copy if its plane is the slab's first or last.
template <int N, int PLANES>
__device__ __forceinline__ void slab_share(Slab<N, PLANES>& L, const SlabPlace<N>& at, int rank, int i, int z,
                                           double value) {
    if (z == at.first && rank > 0) {
        const int li = i - SlabPlace<N>(rank - 1).origin;
        remote_store(remote_address(&L.sol[li & 1][li >> 1], rank - 1), value);
    }
    if (z == at.last - 1 && rank + 1 < kClusterBlocks) {
        const int li = i - SlabPlace<N>(rank + 1).origin;
        remote_store(remote_address(&L.sol[li & 1][li >> 1], rank + 1), value);
    }
}

// The neighbours' sum at local node li (global (x, y)), in the reference's order.
template <int N, int PLANES>
__device__ __forceinline__ double slab_sum(const Slab<N, PLANES>& L, int li, int x, int y) {
    const double* v = L.sol[(li & 1) ^ 1];
    constexpr int none = Slab<N, PLANES>::kSol;
    const double a = v[x > 0 ? (li - 1) >> 1 : none], b = v[x + 1 < N ? (li + 1) >> 1 : none];
    const double c = v[y > 0 ? (li - N) >> 1 : none], d = v[y + 1 < N ? (li + N) >> 1 : none];
    const double e = v[(li - N * N) >> 1], f = v[(li + N * N) >> 1];
    return ((((a + b) + c) + d) + e) + f;
}

template <int N, int PLANES>
__device__ __forceinline__ void slab_relax(Slab<N, PLANES>& L, const SlabPlace<N>& at, int rank, int sweeps) {
    constexpr int NN = N * N;
    const double h2 = (double)(N - 1) * (double)(N - 1);
    for (int phase = 0; phase < 2 * sweeps; ++phase) {
        const int begin = at.first * NN, i0 = begin + ((begin ^ phase) & 1);
        for (int i = i0 + 2 * (int)threadIdx.x; i < at.last * NN; i += 2 * kClusterThreads) {
            const int row = i / N, x = i - row * N, z = row / N, y = row - z * N;
            const int li = i - at.origin, c = li & 1, p = (li >> 1) - at.own;
            const double d = L.diag[c][p];
            if (d > 1.0e-30) {
                const double s = slab_sum(L, li, x, y);
                const double value = divide(__fma_rn(s, h2, L.rhs[c][p]), d, L.inv[c][p]);
                L.sol[c][li >> 1] = value;
                slab_share(L, at, rank, i, z, value);
            }
        }
        cluster_barrier();
    }
}

// Residuals of the slab: out(plane, index in the plane, value).
template <int N, int PLANES, typename Out>
__device__ __forceinline__ void slab_residual(const Slab<N, PLANES>& L, const SlabPlace<N>& at, Out&& out) {
    constexpr int NN = N * N;
    const double h2 = (double)(N - 1) * (double)(N - 1);
    for (int i = at.first * NN + (int)threadIdx.x; i < at.last * NN; i += kClusterThreads) {
        const int row = i / N, x = i - row * N, z = row / N, y = row - z * N;
        const int li = i - at.origin, c = li & 1, p = (li >> 1) - at.own;
        const double s = slab_sum(L, li, x, y);
        out(z, i - z * NN, L.rhs[c][p] - (L.diag[c][p] * L.sol[c][li >> 1] - s * h2));
    }
}

// x += P coarse at every node of the slab (capi.mojo:677-742), coarse(x, y, z) giving the coarse values.
template <int N, int PLANES, typename Coarse>
__device__ __forceinline__ void slab_prolong(Slab<N, PLANES>& L, const SlabPlace<N>& at, int rank, Coarse&& coarse) {
    constexpr int NN = N * N, C = (N + 1) / 2;
    for (int i = at.first * NN + (int)threadIdx.x; i < at.last * NN; i += kClusterThreads) {
        const int row = i / N, x = i - row * N, z = row / N, y = row - z * N;
        const int x0 = x / 2, y0 = y / 2, z0 = z / 2;
        const int x1 = min(x0 + 1, C - 1), y1 = min(y0 + 1, C - 1), z1 = min(z0 + 1, C - 1);
        const double tx = (x & 1) ? 0.5 : 0.0, ty = (y & 1) ? 0.5 : 0.0, tz = (z & 1) ? 0.5 : 0.0;
        // planes z1 beyond the copies are read only with weight 0: keep to z0 there
        const int zb = (z & 1) ? z1 : z0;
        const double c00 = coarse(x0, y0, z0) * (1.0 - tx) + coarse(x1, y0, z0) * tx;
        const double c10 = coarse(x0, y1, z0) * (1.0 - tx) + coarse(x1, y1, z0) * tx;
        const double c01 = coarse(x0, y0, zb) * (1.0 - tx) + coarse(x1, y0, zb) * tx;
        const double c11 = coarse(x0, y1, zb) * (1.0 - tx) + coarse(x1, y1, zb) * tx;
        const double c0 = c00 * (1.0 - ty) + c10 * ty;
        const double c1 = c01 * (1.0 - ty) + c11 * ty;
        const int li = i - at.origin, c = li & 1;
        const double value = L.sol[c][li >> 1] + (c0 * (1.0 - tz) + c1 * tz);
        L.sol[c][li >> 1] = value;
        slab_share(L, at, rank, i, z, value);
    }
    cluster_barrier();
}

template <int N, int PLANES>
__device__ __forceinline__ void slab_setup(Slab<N, PLANES>& L, const SlabPlace<N>& at,
                                           const double* __restrict__ screen, double pw) {
    constexpr int NN = N * N;
    const double h2 = (double)(N - 1) * (double)(N - 1);
    for (int k = threadIdx.x; k < 2 * (Slab<N, PLANES>::kSol + 1); k += kClusterThreads) (&L.sol[0][0])[k] = 0.0;
    for (int i = at.first * NN + (int)threadIdx.x; i < at.last * NN; i += kClusterThreads) {
        const int row = i / N, x = i - row * N, z = row / N, y = row - z * N;
        const int degree = (x > 0) + (x + 1 < N) + (y > 0) + (y + 1 < N) + (z > 0) + (z + 1 < N);
        const int li = i - at.origin, c = li & 1, p = (li >> 1) - at.own;
        const double d = (double)degree * h2 + pw * screen[i] * h2;
        L.diag[c][p] = d;
        L.inv[c][p] = reciprocal(d);
    }
}

struct ClusterSmem {
    Slab<33, 3> fine;
    Slab<17, 2> mid;
    union {
        double residual33[4][33 * 33];  // planes first - 1 .. last - 1 of this block's slab
        double residual[17 * 17 * 17];  // block 0: of 17^3, then of the levels below
    };
    TailStack<9> below;  // block 0
};

__global__ void __launch_bounds__(kClusterThreads) cluster_kernel(const TailArgs a) {
    extern __shared__ __align__(16) unsigned char raw[];
    ClusterSmem& S = *reinterpret_cast<ClusterSmem*>(raw);
    constexpr int N = 33, M = 17, NN = N * N, MM = M * M;
    const int rank = (int)blockIdx.x, tid = (int)threadIdx.x;
    const SlabPlace<N> at(rank);
    const SlabPlace<M> mid(rank);
    slab_setup(S.fine, at, a.screens[0], a.pw);
    slab_setup(S.mid, mid, a.screens[1], a.pw);
    if (rank == 0 && tid < kTailThreads) tail_setup<9>(S.below, a.screens + 2, a.pw);
    cluster_barrier();  // every copy is zero before values are shared
    for (int i = at.first * NN + tid; i < at.last * NN; i += kClusterThreads) {
        const int li = i - at.origin, c = li & 1;
        S.fine.rhs[c][(li >> 1) - at.own] = 0.0 + a.rhs[i];
        if (!a.zero_start) {
            const double value = a.sol[i];
            S.fine.sol[c][li >> 1] = value;
            slab_share(S.fine, at, rank, i, i / NN, value);
        }
    }
    cluster_barrier();
    for (int cycle = 0; cycle < a.cycles; ++cycle) {
        slab_relax(S.fine, at, rank, a.pre);
        // residual of 33^3; the slab's last plane also to the block above, which restricts from it.  17^3 starts at
        // zero, its copies too, before the barrier that lets the neighbours share
        slab_residual(S.fine, at, [&](int z, int k, double r) {
            S.residual33[z - at.first + 1][k] = r;
            if (z == at.last - 1 && rank + 1 < kClusterBlocks) remote_store(remote_address(&S.residual33[0][k], rank + 1), r);
        });
        for (int k = tid; k < 2 * (Slab<M, 2>::kSol + 1); k += kClusterThreads) (&S.mid.sol[0][0])[k] = 0.0;
        cluster_barrier();
        for (int i = mid.first * MM + tid; i < mid.last * MM; i += kClusterThreads) {  // capi.mojo:557-673
            const int row = i / M, x = i - row * M, z = row / M, y = row - z * M;
            double sum = 0.0, weight = 0.0;
#pragma unroll 1
            for (int oz = -1; oz <= 1; ++oz)
#pragma unroll
                for (int oy = -1; oy <= 1; ++oy)
#pragma unroll
                    for (int ox = -1; ox <= 1; ++ox) {
                        const int zz = 2 * z + oz, yy = 2 * y + oy, xx = 2 * x + ox;
                        const double w = (oz ? 1.0 : 2.0) * (oy ? 1.0 : 2.0) * (ox ? 1.0 : 2.0);
                        if ((unsigned)zz < N && (unsigned)yy < N && (unsigned)xx < N) {
                            sum += S.residual33[zz - at.first + 1][yy * N + xx] * w;
                            weight += w;
                        }
                    }
            const int li = i - mid.origin;
            S.mid.rhs[li & 1][(li >> 1) - mid.own] = sum / weight;
        }
        __syncthreads();
        slab_relax(S.mid, mid, rank, a.pre);
        // every block is past its restriction: block 0's residual buffer is free for 17^3's
        slab_residual(S.mid, mid, [&](int z, int k, double r) {
            remote_store(remote_address(&S.residual[z * MM + k], 0), r);
        });
        cluster_barrier();
        if (rank == 0 && tid < kTailThreads) {
            tail_restrict<M, 9>(S.residual, S.below.level);
            tail_barrier<M>();
            if (tid < Tail<9>::kThreads) tail_cycle<9>(S.below, S.residual, a.pre, a.post);
        }
        cluster_barrier();
        slab_prolong(S.mid, mid, rank, [&](int x, int y, int z) {
            const int j = (z * 9 + y) * 9 + x;
            return remote_load(remote_address(&S.below.level.sol[j & 1][j >> 1], 0));
        });
        slab_relax(S.mid, mid, rank, a.post);
        slab_prolong(S.fine, at, rank, [&](int x, int y, int z) {
            const int li = (z * M + y) * M + x - mid.origin;
            return S.mid.sol[li & 1][li >> 1];
        });
        slab_relax(S.fine, at, rank, a.post);
    }
    for (int i = at.first * NN + tid; i < at.last * NN; i += kClusterThreads) {
        const int li = i - at.origin;
        a.sol[i] = S.fine.sol[li & 1][li >> 1];
    }
    cluster_barrier();  // no block leaves while another may still store to it
}

static int launch_cluster(const TailArgs& a, cudaStream_t s, bool only_ask, bool* possible) {
    static_assert(sizeof(ClusterSmem) <= 227 * 1024, "one block's shared memory");
    const void* kernel = (const void*)cluster_kernel;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(kClusterBlocks);
    config.blockDim = dim3(kClusterThreads);
    config.dynamicSmemBytes = sizeof(ClusterSmem);
    config.stream = s;
    cudaLaunchAttribute attribute = {};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = kClusterBlocks;
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClusterSmem));
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (only_ask) {
        int clusters = 0;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &config);
        *possible = e == cudaSuccess && clusters >= 1;
        if (e != cudaSuccess) (void)cudaGetLastError();
        return PB_OK;
    }
    PB_CHECK_CUDA(e, "cluster_kernel attributes");
    void* args[] = {const_cast<TailArgs*>(&a)};
    PB_CHECK_CUDA(cudaLaunchKernelExC(&config, kernel, args), "cluster_kernel");
    PB_CHECK_LAUNCH("cluster_kernel");
    return PB_OK;
}

// Whether this device can place a cluster of 16 such blocks (asked once per device).  The checked
// build answers no: its tests are the ones of the form for devices that cannot, 33^3 colour-split
// over the one-block tail from 17^3.
static bool cluster_possible() {
#ifdef PB_CHECKED
    return false;
#endif
    static std::mutex mu;
    static std::map<int, bool> known;
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(device);
    if (it == known.end()) {
        bool possible = false;
        (void)launch_cluster(TailArgs{}, nullptr, true, &possible);
        it = known.emplace(device, possible).first;
    }
    return it->second;
}

static bool tail_side(int64_t n) { return n == 17 || n == 9 || n == 5 || n == 3 || (n == 33 && cluster_possible()); }

template <int N>
static int launch_tail_n(const TailArgs& a, cudaStream_t s) {
    static_assert(sizeof(TailSmem<N>) <= 227 * 1024, "one block's shared memory");
    PB_CHECK_CUDA(cudaFuncSetAttribute(tail_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(TailSmem<N>)),
                  "tail_kernel attributes");
    tail_kernel<N><<<1, kTailThreads, sizeof(TailSmem<N>), s>>>(a);
    PB_CHECK_LAUNCH("tail_kernel");
    return PB_OK;
}

static int launch_tail(int64_t n, const TailArgs& a, cudaStream_t s) {
    switch (n) {
        case 33: return launch_cluster(a, s, false, nullptr);
        case 17: return launch_tail_n<17>(a, s);
        case 9: return launch_tail_n<9>(a, s);
        case 5: return launch_tail_n<5>(a, s);
        case 3: return launch_tail_n<3>(a, s);
    }
    return fail(PB_ERR_INVALID, "cycle: no tail of side %lld", (long long)n);
}

// ---- the larger levels: colour-split grids -------------------------------------------
//
// A one-colour pass over the reference's dense layout touches every 32-byte sector
// of the iterate, right-hand side and screen for half of the nodes: 32 bytes of
// traffic per node and pass.  Here a level keeps its two colours apart: colour c
// of row (y, z) is stored compactly, entry i being node x = 2i + ((y + z + c) & 1).
// A node's six neighbours are of the other colour: the entry i of its own row and
// of rows y +- 1 and planes z +- 1, and entry i - 1 (even x) or i + 1 (odd x) of
// its own row.  One zero row around every plane, one zero plane below and above
// and at least one zero entry after every row stand for absent neighbours, so the
// sum needs no test.  A pass reads the other colour, its own right-hand side and a
// byte per two nodes, and writes its own colour: 12.5 bytes per node of the grid.
// The byte says whether either node has screening; only then is the dense screen
// read (2 % of the nodes at 257^3) and the general division taken.  On the finest
// level it also says whether either right-hand side is not zero, and the pass moves
// 8.5 bytes per node.  Without
// screening the diagonal is 3 h^-2 .. 6 h^-2, and with y = RN(1 / d) off by at most
// 2^-54 relative for these (h^-2 a power of two), a y is within one ulp of the
// quotient and a single correction of Markstein's (above) rounds it correctly.
// Measured on B200 at 257^3, one colour of one sweep: dense 110 us, split 42 us
// (126 MB of DRAM traffic; latency-bound: half of the warps resident, 58 % of issue
// slots); a whole V(3,3) cycle 2.0 -> 1.0 ms.
struct Split {
    int n, pitch, groups;  // entries per row (even), pairs of entries per row
    uint32_t plane, count;  // entries per plane and per colour, ghosts included (n <= 1025: below 2^31)
    explicit __host__ __device__ Split(int side)
        : n(side), pitch((side + 1) / 2 + 1), groups(pitch / 2), plane((uint32_t)(side + 2) * pitch),
          count((uint32_t)(side + 2) * plane) {}
    __host__ __device__ __forceinline__ uint32_t at(int i, int y, int z) const {
        return (uint32_t)(z + 1) * plane + (uint32_t)(y + 1) * pitch + i;
    }
    // entry of node (x, y, z) in its colour's array
    __host__ __device__ __forceinline__ uint32_t node(int x, int y, int z) const { return at(x >> 1, y, z); }
};

// Of a pair of entries: either node has screening; either right-hand side is not zero (set everywhere below the
// finest level, whose right-hand side is zero but for the nodes around the samples).
constexpr uint8_t kScreened = 1, kSource = 2;

struct SplitLevel {
    double* x[2];          // iterate by colour
    double* f[2];          // right-hand side by colour
    uint8_t* flags[2];     // per pair of entries: kScreened, kSource
    const double* screen;  // dense
};

// Quotient constants of the unscreened diagonals: y[k] = RN(1 / (k h^-2)).
struct Inverse {
    double h2, pw, d6, y6, y5, y4, y3;
    explicit Inverse(int n, double point_weight) {
        const double h = (double)(n - 1);
        h2 = h * h;
        pw = point_weight;
        d6 = 6.0 * h2;
        y6 = 1.0 / d6;
        y5 = 1.0 / (5.0 * h2);
        y4 = 1.0 / (4.0 * h2);
        y3 = 1.0 / (3.0 * h2);
    }
};

__device__ __forceinline__ bool plain_exponent(double a) {  // |a| in [2^-900, 2^901)
    return ((uint32_t)__double2hiint(a) & 0x7ff00000u) - (123u << 20) <= (1800u << 20);
}

// a / d by one correction of a y (above).
__device__ __forceinline__ double corrected(double a, double d, double y) {
    const double q = a * y;
    return __fma_rn(__fma_rn(-d, q, a), y, q);
}

__device__ __forceinline__ double degree_inverse(int degree, const Inverse& v) {
    return degree == 6 ? v.y6 : degree == 5 ? v.y5 : degree == 4 ? v.y4 : v.y3;
}

// The quotients of a pair of entries without screening.  `inner`: the pair's row is inside the y and z faces (the
// same for nearly every warp), where only the first node can have fewer than six neighbours (x_face: at x = 0 or
// n - 1; n - 1 is a multiple of four, so the second never lies there).
__device__ __forceinline__ double2 unscreened_pair(double a0, double a1, bool inner, bool x_face, int degree_yz,
                                                   const Inverse& v) {
    double d0 = v.d6, y0 = v.y6, d1 = v.d6, y1 = v.y6;
    if (inner) {
        if (x_face) {
            d0 = 5.0 * v.h2;
            y0 = v.y5;
        }
    } else {
        const int k0 = degree_yz + (x_face ? 1 : 2), k1 = degree_yz + 2;
        d0 = (double)k0 * v.h2;
        y0 = degree_inverse(k0, v);
        d1 = (double)k1 * v.h2;
        y1 = degree_inverse(k1, v);
    }
    double2 q = make_double2(corrected(a0, d0, y0), corrected(a1, d1, y1));
    if (!plain_exponent(a0) || !plain_exponent(a1)) {
        if (!plain_exponent(a0)) q.x = a0 == 0.0 ? a0 : a0 / d0;
        if (!plain_exponent(a1)) q.y = a1 == 0.0 ? a1 : a1 / d1;
    }
    return q;
}

// Level set-up: the iterate (init inside the grid), the right-hand side of the
// finest level split from the dense one (-0.0 as +0.0: the reference's sums start
// from +0.0), zero ghosts everywhere, and the screening bytes.
__global__ void __launch_bounds__(256) split_setup_kernel(Split g, SplitLevel L, const double* __restrict__ rhs,
                                                          double init) {
    const uint32_t total = (uint32_t)(g.n + 2) * (g.n + 2) * g.groups;
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    if (t >= total) return;
    const int k = t % (uint32_t)g.groups, row = t / (uint32_t)g.groups;
    const int y = row % (g.n + 2) - 1, z = row / (g.n + 2) - 1;
    const bool in = (unsigned)y < (unsigned)g.n && (unsigned)z < (unsigned)g.n;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        double v[2] = {0.0, 0.0}, f[2] = {0.0, 0.0};
        bool screened = false, source = !rhs;
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const int x = 4 * k + 2 * m + ((y + z + c) & 1);
            if (in && x < g.n) {
                const int64_t i = ((int64_t)z * g.n + y) * g.n + x;
                v[m] = init;
                if (rhs) f[m] = 0.0 + rhs[i];
                source |= f[m] != 0.0;
                screened |= L.screen[i] != 0.0;
            }
        }
        const uint32_t at = g.at(2 * k, y, z);
        *reinterpret_cast<double2*>(L.x[c] + at) = make_double2(v[0], v[1]);
        *reinterpret_cast<double2*>(L.f[c] + at) = make_double2(f[0], f[1]);
        if (in) L.flags[c][((uint32_t)z * g.n + y) * g.groups + k] = (screened ? kScreened : 0) | (source ? kSource : 0);
    }
}

// The dense iterate: threads flattened over a plane's (x, y), several planes each so that enough loads are in
// flight (one node per thread took 73 us at 257^3).
constexpr int kMergeZ = 8;
__global__ void __launch_bounds__(256) split_merge_kernel(Split g, const double* __restrict__ x0,
                                                          const double* __restrict__ x1, double* __restrict__ out) {
    const uint32_t t = blockIdx.x * 256u + threadIdx.x, n = g.n;
    if (t >= n * n) return;
    const uint32_t y = t / n, x = t - y * n, z0 = blockIdx.y * kMergeZ, z1 = min(n, z0 + kMergeZ);
    uint32_t at = g.node(x, y, z0);
#pragma unroll
    for (uint32_t z = z0; z < z0 + kMergeZ; ++z, at += g.plane)
        if (z < z1) out[((uint64_t)z * n + y) * n + x] = (((x + y + z) & 1) ? x1 : x0)[at];
}

__device__ __forceinline__ double2 pair_at(const double* p, uint32_t i) {
    return *reinterpret_cast<const double2*>(p + i);
}

// One colour of one sweep: own <- from other.  A thread takes two neighbouring
// entries of a row and marches down z with the other colour's planes z - 1, z and
// z + 1 in registers.  ZERO: the other colour is zero (a coarse level's first
// pass).  SPARSE (the finest level): the right-hand side is read only where it is
// not zero, its flag having been read a plane ahead.  Bound by memory latency: five
// blocks per SM (48 registers) measured best.
template <bool ZERO, bool SPARSE>
__global__ void __launch_bounds__(256, 5) split_relax_kernel(Split g, double* __restrict__ own,
                                                             const double* __restrict__ other,
                                                             const double* __restrict__ f,
                                                             const uint8_t* __restrict__ flags,
                                                             const double* __restrict__ screen, Inverse v, int colour,
                                                             int planes) {
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    if (t >= (uint32_t)g.n * g.groups) return;
    const int n = g.n, y = t / (uint32_t)g.groups, k = t - y * g.groups;
    const int z0 = blockIdx.y * planes, z1 = min(n, z0 + planes);
    uint32_t at = g.at(2 * k, y, z0);
    double2 below = make_double2(0.0, 0.0), here = below, above = below;
    if (!ZERO) {
        below = pair_at(other, at - g.plane);
        here = pair_at(other, at);
    }
    const int degree_y = (y > 0) + (y + 1 < n), k_last = (n - 1) / 4 - 1;
    const bool k_face = k == 0 || 4 * k == n - 1;
    int flag_here = SPARSE ? flags[((uint32_t)z0 * n + y) * g.groups + k] : 0;
    for (int z = z0; z < z1; ++z, at += g.plane) {
        const int odd = (y + z + colour) & 1, x = 4 * k + odd;  // nodes x and x + 2
        double s0 = 0.0, s1 = 0.0;
        double2 rhs = make_double2(0.0, 0.0);
        int flag, ahead = 0;
        if (SPARSE) {
            flag = flag_here;
            if (z + 1 < z1) ahead = flags[((uint32_t)(z + 1) * n + y) * g.groups + k];
            if (flag & kSource) rhs = pair_at(f, at);
        } else {
            flag = flags[((uint32_t)z * n + y) * g.groups + k];
            rhs = pair_at(f, at);
        }
        double scr0 = 0.0, scr1 = 0.0;
        if (flag & kScreened) {
            const double* scr = screen + ((int64_t)z * n + y) * n + x;
            if (x < n) scr0 = scr[0];
            if (x + 2 < n) scr1 = scr[2];
        }
        if (!ZERO) {
            above = pair_at(other, at + g.plane);
            const double2 up = pair_at(other, at - g.pitch), down = pair_at(other, at + g.pitch);
            const double outer = other[odd ? at + 2 : at - 1];
            s0 = here.x + (odd ? here.y : outer);
            s1 = here.y + (odd ? outer : here.x);
            s0 += up.x;
            s1 += up.y;
            s0 += down.x;
            s1 += down.y;
            s0 += below.x;
            s1 += below.y;
            s0 += above.x;
            s1 += above.y;
        }
        const double a0 = __fma_rn(s0, v.h2, rhs.x), a1 = __fma_rn(s1, v.h2, rhs.y);  // s h2 is exact: h2 = 4^k
        const int degree = degree_y + (z > 0) + (z + 1 < n);
        const bool x_face = k_face && !odd;
        double2 q;
        if (!(flag & kScreened)) {
            q = unscreened_pair(a0, a1, degree == 4, x_face, degree, v);
        } else {
            const int d0 = degree + (x_face ? 1 : 2), d1 = degree + 2;
            const double e0 = (double)d0 * v.h2 + v.pw * scr0 * v.h2, e1 = (double)d1 * v.h2 + v.pw * scr1 * v.h2;
            q.x = e0 > 1.0e-30 ? a0 / e0 : own[at];
            q.y = e1 > 1.0e-30 ? a1 / e1 : own[at + 1];
        }
        if (k >= k_last) {  // the row's zero entries
            if (x >= n) q.x = 0.0;
            if (x + 2 >= n) q.y = 0.0;
        }
        *reinterpret_cast<double2*>(own + at) = q;
        below = here;
        here = above;
        flag_here = ahead;
    }
}

// r = rhs - A x (capi.mojo:413-553) at the four nodes 4k .. 4k + 3 of row y, plane by plane down z, with both
// colours' planes z - 1, z and z + 1 in registers.
template <bool SPARSE>
struct ResidualMarch {
    const Split g;
    const SplitLevel& L;
    const Inverse& v;
    const int y, k, degree_y;
    uint32_t at;
    double2 below[2], here[2], above[2];  // by colour
    int flag[2];

    __device__ __forceinline__ ResidualMarch(const Split& split, const SplitLevel& level, const Inverse& inverse,
                                             int row, int group, int z0)
        : g(split), L(level), v(inverse), y(row), k(group), degree_y((row > 0) + (row + 1 < split.n)),
          at(split.at(2 * group, row, z0)) {
        below[0] = pair_at(L.x[0], at - g.plane);
        below[1] = pair_at(L.x[1], at - g.plane);
        here[0] = pair_at(L.x[0], at);
        here[1] = pair_at(L.x[1], at);
        read_flags(z0);
    }

    __device__ __forceinline__ void read_flags(int z) {
        const uint32_t i = ((uint32_t)z * g.n + y) * g.groups + k;
        flag[0] = L.flags[0][i];
        flag[1] = L.flags[1][i];
    }

    __device__ __forceinline__ void step(int z, double (&r)[4]) {
        const int n = g.n, odd = (y + z) & 1, degree = degree_y + (z > 0) + (z + 1 < n);
        above[0] = pair_at(L.x[0], at + g.plane);
        above[1] = pair_at(L.x[1], at + g.plane);
        const uint32_t row = (uint32_t)z * n + y;
        const int now[2] = {flag[0], flag[1]};
        if (z + 1 < n) read_flags(z + 1);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int first = odd ^ c, x = 4 * k + first;  // colour c: nodes x and x + 2
            const double* o = L.x[1 - c];
            const double2 up = pair_at(o, at - g.pitch), down = pair_at(o, at + g.pitch);
            double2 f = make_double2(0.0, 0.0);
            if (!SPARSE || (now[c] & kSource)) f = pair_at(L.f[c], at);
            const double outer = o[first ? at + 2 : at - 1];
            const double2 mid = here[1 - c];
            double s0 = mid.x + (first ? mid.y : outer), s1 = mid.y + (first ? outer : mid.x);
            s0 += up.x;
            s1 += up.y;
            s0 += down.x;
            s1 += down.y;
            s0 += below[1 - c].x;
            s1 += below[1 - c].y;
            s0 += above[1 - c].x;
            s1 += above[1 - c].y;
            double e0 = (double)(degree + (x > 0) + (x + 1 < n)) * v.h2, e1 = (double)(degree + 1 + (x + 3 < n)) * v.h2;
            if (now[c] & kScreened) {
                const double* scr = L.screen + (int64_t)row * n + x;
                if (x < n) e0 += v.pw * scr[0] * v.h2;
                if (x + 2 < n) e1 += v.pw * scr[2] * v.h2;
            }
            const double r0 = x < n ? f.x - (e0 * here[c].x - s0 * v.h2) : 0.0;
            const double r1 = x + 2 < n ? f.y - (e1 * here[c].y - s1 * v.h2) : 0.0;
            if (first) {
                r[1] = r0;
                r[3] = r1;
            } else {
                r[0] = r0;
                r[2] = r1;
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            below[c] = here[c];
            here[c] = above[c];
        }
        at += g.plane;
    }
};

// The residual restricted to the next level's right-hand side (capi.mojo:557-673),
// without storing it: a block owns up to kCoarseX x kCoarseY coarse columns and
// marches down z; each fine residual plane over them goes to shared memory once
// (two by parity: one barrier per plane) and is added to the coarse sums it belongs
// to, in the reference's order.  257^3: 115 us (tiles of 34 x 9, 34 x 4 and 18 x 9
// coarse columns 118-124) against 170 for the dense residual and 100 for the dense
// restriction.  SPLIT_OUT: the coarse level is colour-split (else
// dense: the tail's top level).
constexpr int kCoarseX = 34, kCoarseY = 6;  // kCoarseX even: 129 = 4 x 33 coarse columns in four tiles
constexpr int kResGroups = kCoarseX / 2 + 1, kResRows = 2 * kCoarseY + 1, kResPitch = 4 * kResGroups;
constexpr int kRestrictThreads = (kResGroups * kResRows + 31) / 32 * 32;

template <bool SPLIT_OUT, bool SPARSE>
__global__ void __launch_bounds__(kRestrictThreads, 3) split_restrict_kernel(Split g, const SplitLevel L, Inverse v,
                                                                             double* __restrict__ out0,
                                                                             double* __restrict__ out1, int width,
                                                                             int height, int planes) {
    __shared__ __align__(16) double res[2][kResRows * kResPitch];
    const int n = g.n, cn = (n + 1) / 2, tid = threadIdx.x;
    const int X0 = blockIdx.x * width, Y0 = blockIdx.y * height, Z0 = blockIdx.z * planes, Z1 = min(cn, Z0 + planes);
    const int ry = tid / kResGroups, gx = tid - ry * kResGroups;
    const int y = 2 * Y0 - 1 + ry, k = X0 / 2 - 1 + gx;
    const bool slot = ry < kResRows;
    const bool in = ry < 2 * height + 1 && gx < width / 2 + 1 && (unsigned)y < (unsigned)n && (unsigned)k < (unsigned)g.groups;
    const int cy = tid / kCoarseX, cx = tid - cy * kCoarseX, X = X0 + cx, Y = Y0 + cy;
    const bool coarse = cx < width && cy < height && X < cn && Y < cn;
    const double weight_xy = (X > 0 && X + 1 < cn ? 4.0 : 3.0) * (Y > 0 && Y + 1 < cn ? 4.0 : 3.0);
    const Split cg(cn);
    double acc = 0.0;
    const int z0 = max(2 * Z0 - 1, 0), z1 = min(2 * Z1 - 1, n - 1);
    ResidualMarch<SPARSE> march(g, L, v, in ? y : 0, in ? k : 0, z0);
    for (int z = z0; z <= z1; ++z) {
        double* plane = res[z & 1];
        double r[4];
        march.step(z, r);
        if (slot) {
            double2* row = reinterpret_cast<double2*>(plane + ry * kResPitch + 4 * gx);
            row[0] = in ? make_double2(r[0], r[1]) : make_double2(0.0, 0.0);
            row[1] = in ? make_double2(r[2], r[3]) : make_double2(0.0, 0.0);
        }
        __syncthreads();  // the other plane is written again only after the next barrier
        if (!coarse) continue;
        const double* p = plane + (2 * cy + 1) * kResPitch + 2 * cx + 4;
        auto add = [&](double wz) {
#pragma unroll
            for (int oy = -1; oy <= 1; ++oy)
#pragma unroll
                for (int ox = -1; ox <= 1; ++ox)
                    acc += p[oy * kResPitch + ox] * ((ox ? 1.0 : 2.0) * (oy ? 1.0 : 2.0) * wz);
        };
        const int Z = z >> 1;  // even z: its own coarse plane; odd z: the upper half of Z, the lower half of Z + 1
        if (z & 1) add(1.0);
        else add(2.0);
        if ((z & 1) || z == n - 1) {
            if (Z >= Z0) {
                const double value = acc / (weight_xy * (Z > 0 && Z + 1 < cn ? 4.0 : 3.0));
                if (SPLIT_OUT) (((X + Y + Z) & 1) ? out1 : out0)[cg.node(X, Y, Z)] = value;
                else out0[((int64_t)Z * cn + Y) * cn + X] = value;
            }
            acc = 0.0;
            add(1.0);
        }
    }
}

// x += P coarse (capi.mojo:677-742) at the nodes of colour 1 only: the pass that
// follows overwrites every node of colour 0 from those.
template <bool SPLIT_IN>
__global__ void __launch_bounds__(256) split_prolong_kernel(Split g, double* __restrict__ x1,
                                                            const double* __restrict__ c0,
                                                            const double* __restrict__ c1) {
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    if (t >= (uint32_t)g.n * g.n * g.groups) return;
    const int n = g.n, cn = (n + 1) / 2, row = t / (uint32_t)g.groups, k = t - row * g.groups;
    const int y = row % n, z = row / n, odd = (y + z + 1) & 1;
    const Split cg(cn);
    auto at = [&](int X, int Y, int Z) -> double {
        if (X >= cn) return 0.0;  // only for entries outside the grid
        return SPLIT_IN ? (((X + Y + Z) & 1) ? c1 : c0)[cg.node(X, Y, Z)] : c0[((int64_t)Z * cn + Y) * cn + X];
    };
    const int X = 2 * k, Y = y >> 1, Z = z >> 1;  // nodes 4k + odd and 4k + 2 + odd: X and X + 1 (+ 1/2 if odd)
    // a weight 1 - t = 1 leaves a value as it is; halves are exact
    auto in_x = [&](int YY, int ZZ) {
        const double a = at(X, YY, ZZ), b = at(X + 1, YY, ZZ);
        if (!odd) return make_double2(a, b);
        const double c = at(X + 2, YY, ZZ);
        return make_double2(a * 0.5 + b * 0.5, b * 0.5 + c * 0.5);
    };
    auto half = [](double2 a, double2 b) { return make_double2(a.x * 0.5 + b.x * 0.5, a.y * 0.5 + b.y * 0.5); };
    auto in_y = [&](int ZZ) { return (y & 1) ? half(in_x(Y, ZZ), in_x(Y + 1, ZZ)) : in_x(Y, ZZ); };
    const double2 e = (z & 1) ? half(in_y(Z), in_y(Z + 1)) : in_y(Z);
    double2* p = reinterpret_cast<double2*>(x1 + g.at(2 * k, y, z));
    double2 value = *p;
    if (4 * k + odd < n) value.x += e.x;
    if (4 * k + 2 + odd < n) value.y += e.y;
    *p = value;
}

// Per-block sums of the squared residual.
__global__ void __launch_bounds__(256) split_norm_kernel(Split g, const SplitLevel L, Inverse v, int planes,
                                                         double* __restrict__ partial) {
    __shared__ double sums[8];
    const uint32_t t = blockIdx.x * 256u + threadIdx.x;
    double sq = 0.0;
    if (t < (uint32_t)g.n * g.groups) {
        const int y = t / (uint32_t)g.groups, k = t - y * g.groups;
        const int z0 = blockIdx.y * planes, z1 = min(g.n, z0 + planes);
        ResidualMarch<true> march(g, L, v, y, k, z0);
        for (int z = z0; z < z1; ++z) {
            double r[4];
            march.step(z, r);
#pragma unroll
            for (int i = 0; i < 4; ++i) sq += r[i] * r[i];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        double total = 0.0;
        for (int w = 0; w < 8; ++w) total += sums[w];
        partial[blockIdx.y * gridDim.x + blockIdx.x] = total;
    }
}

__global__ void __launch_bounds__(256) norm_finish_kernel(const double* __restrict__ partial, int count,
                                                          double* __restrict__ norm) {
    __shared__ double sums[8];
    double v = 0.0;
    for (int i = threadIdx.x; i < count; i += 256) v += partial[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double total = 0.0;
        for (int w = 0; w < 8; ++w) total += sums[w];
        *norm = sqrt(total);
    }
}

static int tiles(int items, int most) { return (items + most - 1) / most; }

constexpr int kNormPlanes = 8;
static dim3 norm_grid(const Split& g) { return dim3(tiles(g.n * g.groups, 256), tiles(g.n, kNormPlanes)); }
static int norm_blocks(const Split& g) { return norm_grid(g).x * norm_grid(g).y; }

// Planes a block of the relaxation marches.  257^3: 1 plane 61 us, 2: 51, 4: 48, 6: 47, 8: 48, 16: 51; 129^3: 2 or
// 4: 8.3, 1: 10.3, 8: 12.4; smaller levels are one wave of latency whatever the split, so one plane each.  Whole
// cycles: 513^3 4 planes 6.19 ms, 6: 6.15, 8: 6.19, 16: 6.53; 1025^3 4: 47.8, 6: 46.9, 12: 45.8, 24: 46.5.
static int relax_planes(int n) { return n >= 257 ? 6 : n >= 129 ? 4 : 1; }

template <bool ZERO, bool SPARSE>
static int launch_split_relax(const SplitLevel& L, int n, double pw, int colour, cudaStream_t s) {
    const Split g(n);
    const int planes = relax_planes(n);
    split_relax_kernel<ZERO, SPARSE><<<dim3(tiles(n * g.groups, 256), tiles(n, planes)), 256, 0, s>>>(
        g, L.x[colour], L.x[1 - colour], L.f[colour], L.flags[colour], L.screen, Inverse(n, pw), colour, planes);
    PB_CHECK_LAUNCH("split_relax_kernel");
    return PB_OK;
}

static int launch_split_sweeps(const SplitLevel& L, int n, double pw, int sweeps, bool finest, bool from_zero,
                               cudaStream_t s) {
    for (int k = 0; k < 2 * sweeps; ++k)
        PB_TRY(finest                ? (launch_split_relax<false, true>(L, n, pw, k & 1, s))
               : k == 0 && from_zero ? (launch_split_relax<true, false>(L, n, pw, 0, s))
                                     : (launch_split_relax<false, false>(L, n, pw, k & 1, s)));
    return PB_OK;
}

static int launch_split_restrict(const SplitLevel& L, int n, double pw, bool finest, const SplitLevel& below,
                                 bool split_below, cudaStream_t s) {
    const Split g(n);
    const int cn = (n + 1) / 2, width = (tiles(cn, tiles(cn, kCoarseX)) + 1) / 2 * 2, height = tiles(cn, tiles(cn, kCoarseY));
    const int planes = cn >= 129 ? 8 : cn >= 65 ? 4 : 1;
    const dim3 grid(tiles(cn, width), tiles(cn, height), tiles(cn, planes));
    const Inverse v(n, pw);
    auto kernel = split_below ? (finest ? split_restrict_kernel<true, true> : split_restrict_kernel<true, false>)
                              : (finest ? split_restrict_kernel<false, true> : split_restrict_kernel<false, false>);
    kernel<<<grid, kRestrictThreads, 0, s>>>(g, L, v, below.f[0], below.f[1], width, height, planes);
    PB_CHECK_LAUNCH("split_restrict_kernel");
    return PB_OK;
}

static int launch_split_prolong(const SplitLevel& L, int n, const SplitLevel& below, bool split_below,
                                cudaStream_t s) {
    const Split g(n);
    const unsigned blocks = blocks_for((int64_t)n * n * g.groups, 256);
    if (split_below) split_prolong_kernel<true><<<blocks, 256, 0, s>>>(g, L.x[1], below.x[0], below.x[1]);
    else split_prolong_kernel<false><<<blocks, 256, 0, s>>>(g, L.x[1], below.x[0], nullptr);
    PB_CHECK_LAUNCH("split_prolong_kernel");
    return PB_OK;
}

static int check_sides(int64_t levels, const int64_t* sides, const char* what) {
    if (levels < 1 || levels > 16 || !sides) return fail(PB_ERR_INVALID, "%s: bad levels", what);
    for (int64_t l = 0; l < levels; ++l)
        if (sides[l] != (l + 1 < levels ? 2 * sides[l + 1] - 1 : 3) || sides[l] > 1025)
            return fail(PB_ERR_INVALID, "%s: sides must halve from at most 1025 down to 3", what);
    return PB_OK;
}

// Level l of the caller's table: (iterate, right-hand side, screening bytes, dense screen).
static SplitLevel level_of(void* const* grids, int64_t l, int64_t n) {
    SplitLevel L = {};
    L.x[0] = (double*)grids[4 * l];
    L.f[0] = (double*)grids[4 * l + 1];
    L.screen = (const double*)grids[4 * l + 3];
    if (!tail_side(n)) {
        const Split g((int)n);
        L.x[1] = L.x[0] + g.count;
        L.f[1] = L.f[0] + g.count;
        L.flags[0] = (uint8_t*)grids[4 * l + 2];
        L.flags[1] = L.flags[0] + (size_t)n * n * g.groups;
    }
    return L;
}

static int check_grids(int64_t levels, const int64_t* sides, void* const* grids, const char* what) {
    PB_TRY(check_sides(levels, sides, what));
    if (!grids) return fail(PB_ERR_INVALID, "%s: null grids", what);
    int64_t top = 0;
    while (!tail_side(sides[top])) ++top;
    for (int64_t l = 0; l < levels; ++l) {
        if (!grids[4 * l + 3] || (l <= top && (!grids[4 * l] || !grids[4 * l + 1])) || (l < top && !grids[4 * l + 2]))
            return fail(PB_ERR_INVALID, "%s: null grid", what);
        if (l < top && (((uintptr_t)grids[4 * l] | (uintptr_t)grids[4 * l + 1]) & 15))
            return fail(PB_ERR_INVALID, "%s: grids must be 16-byte aligned", what);
    }
    return PB_OK;
}

}  // namespace cycle64
}  // namespace pb

using namespace pb;

// Sizes of one level of pb_vcycles_f64's hierarchy: doubles of its iterate (and
// of its right-hand side), bytes of its screening flags.  Sides <= 17 are dense, and so is 33
// where the current device can place a cluster of 16 blocks.
extern "C" int pb_vcycle_level_size(int64_t n, int64_t* doubles, int64_t* flag_bytes) {
    if (n < 3 || n > 1025 || !doubles || !flag_bytes) return fail(PB_ERR_INVALID, "vcycle level size: bad args");
    if (cycle64::tail_side(n)) {
        *doubles = n * n * n;
        *flag_bytes = 0;
    } else {
        const cycle64::Split g((int)n);
        *doubles = 2 * (int64_t)g.count;
        *flag_bytes = 2 * n * n * g.groups;
    }
    return PB_OK;
}

// Prepares the levels for pb_vcycles_f64: the finest iterate at `init`, the
// finest right-hand side from the dense `rhs`, ghosts and flags of every level.
extern "C" int pb_vcycle_setup_f64(int64_t levels, const int64_t* sides, void* const* grids, const double* rhs,
                                   double init, void* stream) {
    using namespace pb::cycle64;
    PB_TRY(check_grids(levels, sides, grids, "vcycle setup"));
    if (!rhs) return fail(PB_ERR_INVALID, "vcycle setup: null rhs");
    cudaStream_t s = (cudaStream_t)stream;
    for (int64_t l = 0; l < levels && !tail_side(sides[l]); ++l) {
        const Split g((int)sides[l]);
        const int64_t items = (int64_t)(g.n + 2) * (g.n + 2) * g.groups;
        split_setup_kernel<<<blocks_for(items, 256), 256, 0, s>>>(g, level_of(grids, l, sides[l]), l ? nullptr : rhs,
                                                                  l ? 0.0 : init);
        PB_CHECK_LAUNCH("split_setup_kernel");
    }
    if (tail_side(sides[0])) {
        const int64_t count = sides[0] * sides[0] * sides[0];
        PB_TRY(pb_fill_f64((double*)grids[0], count, init, stream));
        PB_CHECK_CUDA(cudaMemcpyAsync(grids[1], rhs, count * sizeof(double), cudaMemcpyDeviceToDevice, s),
                      "vcycle setup rhs");
    }
    return PB_OK;
}

// The finest iterate, dense.
extern "C" int pb_vcycle_field_f64(int64_t n, const double* iterate, double* field, void* stream) {
    using namespace pb::cycle64;
    if (n < 3 || n > 1025 || !iterate || !field) return fail(PB_ERR_INVALID, "vcycle field: bad args");
    cudaStream_t s = (cudaStream_t)stream;
    if (tail_side(n)) {
        PB_CHECK_CUDA(cudaMemcpyAsync(field, iterate, n * n * n * sizeof(double), cudaMemcpyDeviceToDevice, s),
                      "vcycle field");
        return PB_OK;
    }
    const Split g((int)n);
    split_merge_kernel<<<dim3(blocks_for(n * n, 256), (unsigned)((n + kMergeZ - 1) / kMergeZ)), 256, 0, s>>>(
        g, iterate, iterate + g.count, field);
    PB_CHECK_LAUNCH("split_merge_kernel");
    return PB_OK;
}

extern "C" size_t pb_vcycle_workspace_size(int64_t n) {
    if (n < 3 || n > 1025) return 256;
    if (cycle64::tail_side(n)) return (size_t)(n * n * n) * sizeof(double) + pb_residual_workspace_size(n) + 512;
    return (size_t)cycle64::norm_blocks(cycle64::Split((int)n)) * sizeof(double) + 256;
}

// `cycles` V(pre, post) cycles of the FP64 multigrid (core.py:141-193) on a
// hierarchy of sides 2^k + 1, finest first, halving down to 3.  grids: per level
// (iterate, right-hand side, screening flags, dense screen), prepared by
// pb_vcycle_setup_f64; levels below the first dense one (pb_vcycle_level_size) need only the screen.
// norm (may be null): the finest level's ||rhs - A x||_2 after the last cycle.
extern "C" int pb_vcycles_f64(int64_t levels, const int64_t* sides, void* const* grids, double point_weight,
                              int64_t pre, int64_t post, int64_t cycles, double* norm, void* workspace,
                              size_t workspace_bytes, void* stream) {
    using namespace pb::cycle64;
    PB_TRY(check_grids(levels, sides, grids, "vcycles"));
    if (pre < 1 || post < 1 || cycles < 0 || !(point_weight >= 0.0)) return fail(PB_ERR_INVALID, "vcycles: bad args");
    if (norm && (!workspace || workspace_bytes < pb_vcycle_workspace_size(sides[0])))
        return fail(PB_ERR_WORKSPACE, "vcycles: workspace needs %zu bytes", pb_vcycle_workspace_size(sides[0]));
    cudaStream_t s = (cudaStream_t)stream;
    SplitLevel level[16];
    int64_t top = levels;  // first level of the tail
    for (int64_t l = levels - 1; l >= 0; --l) {
        level[l] = level_of(grids, l, sides[l]);
        if (tail_side(sides[l])) top = l;
    }
    TailArgs tail = {};
    for (int64_t l = top; l < levels; ++l) tail.screens[l - top] = level[l].screen;
    tail.rhs = level[top].f[0];
    tail.sol = level[top].x[0];
    tail.pw = point_weight;
    tail.pre = (int)pre;
    tail.post = (int)post;
    tail.zero_start = top > 0;
    tail.cycles = top > 0 ? 1 : (int)cycles;
    if (top == 0) {
        PB_TRY(launch_tail(sides[0], tail, s));
    } else {
        for (int64_t c = 0; c < cycles; ++c) {
            for (int64_t l = 0; l < top; ++l) {
                const int n = (int)sides[l];
                PB_TRY(launch_split_sweeps(level[l], n, point_weight, (int)pre, l == 0, true, s));
                PB_TRY(launch_split_restrict(level[l], n, point_weight, l == 0, level[l + 1], l + 1 < top, s));
            }
            PB_TRY(launch_tail(sides[top], tail, s));
            for (int64_t l = top - 1; l >= 0; --l) {
                const int n = (int)sides[l];
                PB_TRY(launch_split_prolong(level[l], n, level[l + 1], l + 1 < top, s));
                PB_TRY(launch_split_sweeps(level[l], n, point_weight, (int)post, l == 0, false, s));
            }
        }
    }
    if (!norm) return PB_OK;
    if (top == 0) {
        const int64_t n = sides[0];
        const size_t residual = (size_t)(n * n * n) * sizeof(double) + 255 & ~(size_t)255;
        return pb_residual_f64(level[0].x[0], level[0].f[0], level[0].screen, (double*)workspace, n, point_weight, norm,
                               (char*)workspace + residual, workspace_bytes - residual, stream);
    }
    const Split g((int)sides[0]);
    double* partial = (double*)workspace;
    split_norm_kernel<<<norm_grid(g), 256, 0, s>>>(
        g, level[0], Inverse(g.n, point_weight), kNormPlanes, partial);
    PB_CHECK_LAUNCH("split_norm_kernel");
    norm_finish_kernel<<<1, 256, 0, s>>>(partial, norm_blocks(g), norm);
    PB_CHECK_LAUNCH("norm_finish_kernel");
    return PB_OK;
}
