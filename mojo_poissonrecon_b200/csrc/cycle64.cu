// One whole FP64 V-cycle of the reference per call (core.py:141-193), bit-exact.
//
// Every node update here computes what stencil64.cu's kernels compute, in the
// same order (-fmad=false): s = ((((x- + x+) + y-) + y+) + z-) + z+ with absent
// neighbours adding +0.0 (a sum that starts from +0.0 never becomes -0.0, so
// adding +0.0 changes no bit), then (rhs + s h^-2) / diagonal.
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
// and 3 run on the first 416, 96 and 32 threads (their nodes of one colour)
// with named barriers of that many threads.  Measured on B200: a depth-5
// reconstruction of 2,000 points (five cycles) 3.56 -> 1.21 ms, 13,337 points
// at depth 6 (four cycles) 3.38 -> 1.48 ms.
constexpr int kTailThreads = 1024;

template <int N>
struct Tail {
    static constexpr int kNodes = N * N * N;
    static constexpr int kHalf = (N + 1) / 2;
    static constexpr int kItems = kHalf * N * N;  // candidates of one colour
    static constexpr int kThreads = N >= 17 ? kTailThreads : N == 9 ? 416 : N == 5 ? 96 : 32;
    double sol[kNodes + 1];  // the last entry stays +0.0: an absent neighbour
    double rhs[kNodes];
    double diag[kNodes];
    double inv[kNodes];
};

template <int N>
__device__ __forceinline__ void tail_barrier() {
    if (N == 3) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"n"(N >= 17 ? 1 : N == 9 ? 2 : 3), "n"(Tail<N>::kThreads) : "memory");
}

// The six neighbours' slots of node (x, y, z), absent ones at the zero entry.
template <int N>
struct Around {
    int at[6];
    __device__ __forceinline__ Around(int x, int y, int z) {
        const int i = (z * N + y) * N + x, none = N * N * N;
        at[0] = x > 0 ? i - 1 : none;
        at[1] = x + 1 < N ? i + 1 : none;
        at[2] = y > 0 ? i - N : none;
        at[3] = y + 1 < N ? i + N : none;
        at[4] = z > 0 ? i - N * N : none;
        at[5] = z + 1 < N ? i + N * N : none;
    }
    __device__ __forceinline__ double sum(const double* v) const {
        return ((((v[at[0]] + v[at[1]]) + v[at[2]]) + v[at[3]]) + v[at[4]]) + v[at[5]];
    }
};

template <int N>
__device__ __forceinline__ void tail_update(Tail<N>& L, int i, const Around<N>& a, double h2) {
    const double s = 0.0 + a.sum(L.sol), d = L.diag[i];
    if (d > 1.0e-30) L.sol[i] = divide(L.rhs[i] + s * h2, d, L.inv[i]);
}

// Sweeps of level N; every thread below kThreads takes part.
template <int N>
__device__ __forceinline__ void tail_relax(Tail<N>& L, int sweeps) {
    const double h2 = (double)(N - 1) * (double)(N - 1);
    const int tid = threadIdx.x;
    if constexpr (N <= 5) {  // at most one node of each colour per thread: addresses once
        const int k = tid % Tail<N>::kHalf, row = tid / Tail<N>::kHalf, y = row % N, z = row / N;
        const int xa = ((y + z) & 1) + 2 * k, xb = ((y + z + 1) & 1) + 2 * k;
        const bool ok = tid < Tail<N>::kItems, oka = ok && xa < N, okb = ok && xb < N;
        const Around<N> a(oka ? xa : 0, oka ? y : 0, oka ? z : 0), b(okb ? xb : 0, okb ? y : 0, okb ? z : 0);
        const int ia = (z * N + y) * N + xa, ib = (z * N + y) * N + xb;
        for (int it = 0; it < sweeps; ++it) {
            if (oka) tail_update<N>(L, ia, a, h2);
            tail_barrier<N>();
            if (okb) tail_update<N>(L, ib, b, h2);
            tail_barrier<N>();
        }
    } else {
        for (int phase = 0; phase < 2 * sweeps; ++phase) {
            for (int t = tid; t < Tail<N>::kItems; t += Tail<N>::kThreads) {
                const int k = t % Tail<N>::kHalf, row = t / Tail<N>::kHalf, y = row % N, z = row / N;
                const int x = ((y + z + phase) & 1) + 2 * k;
                if (x < N) tail_update<N>(L, (z * N + y) * N + x, Around<N>(x, y, z), h2);
            }
            tail_barrier<N>();
        }
    }
}

template <int N>
__device__ __forceinline__ void tail_residual(const Tail<N>& L, double* __restrict__ res) {
    const double h2 = (double)(N - 1) * (double)(N - 1);
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += Tail<N>::kThreads) {
        const int x = i % N, y = (i / N) % N, z = i / (N * N);
        const double s = 0.0 + Around<N>(x, y, z).sum(L.sol);
        res[i] = L.rhs[i] - (L.diag[i] * L.sol[i] - s * h2);
    }
}

// capi.mojo:557-673 from the fine residual; the coarse iterate starts at zero.
template <int N, int C>
__device__ __forceinline__ void tail_restrict(const double* __restrict__ res, Tail<C>& L) {
    for (int i = threadIdx.x; i < Tail<C>::kNodes; i += Tail<N>::kThreads) {
        const int x = i % C, y = (i / C) % C, z = i / (C * C);
        double sum = 0.0, weight = 0.0;
#pragma unroll
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
        L.rhs[i] = sum / weight;
        L.sol[i] = 0.0;
    }
}

// capi.mojo:677-742
template <int N, int C>
__device__ __forceinline__ void tail_prolong(Tail<N>& L, const Tail<C>& K) {
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += Tail<N>::kThreads) {
        const int x = i % N, y = (i / N) % N, z = i / (N * N);
        const int x0 = x / 2, y0 = y / 2, z0 = z / 2;
        const int x1 = min(x0 + 1, C - 1), y1 = min(y0 + 1, C - 1), z1 = min(z0 + 1, C - 1);
        const double tx = (x & 1) ? 0.5 : 0.0, ty = (y & 1) ? 0.5 : 0.0, tz = (z & 1) ? 0.5 : 0.0;
        const double* c = K.sol;
        auto at = [&](int xx, int yy, int zz) { return c[(zz * C + yy) * C + xx]; };
        const double c00 = at(x0, y0, z0) * (1.0 - tx) + at(x1, y0, z0) * tx;
        const double c10 = at(x0, y1, z0) * (1.0 - tx) + at(x1, y1, z0) * tx;
        const double c01 = at(x0, y0, z1) * (1.0 - tx) + at(x1, y0, z1) * tx;
        const double c11 = at(x0, y1, z1) * (1.0 - tx) + at(x1, y1, z1) * tx;
        const double c0 = c00 * (1.0 - ty) + c10 * ty;
        const double c1 = c01 * (1.0 - ty) + c11 * ty;
        L.sol[i] += c0 * (1.0 - tz) + c1 * tz;
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
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += kTailThreads) {
        const int x = i % N, y = (i / N) % N, z = i / (N * N);
        const int degree = (x > 0) + (x + 1 < N) + (y > 0) + (y + 1 < N) + (z > 0) + (z + 1 < N);
        const double d = (double)degree * h2 + pw * screen[i] * h2;
        S.level.diag[i] = d;
        S.level.inv[i] = reciprocal(d);
    }
    if (threadIdx.x == 0) S.level.sol[Tail<N>::kNodes] = 0.0;
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
    const double* screens[4];  // top level first
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
        S.stack.level.rhs[i] = a.rhs[i];
        S.stack.level.sol[i] = a.zero_start ? 0.0 : a.sol[i];
    }
    __syncthreads();
    for (int c = 0; c < a.cycles; ++c) {
        if (threadIdx.x < Tail<N>::kThreads) tail_cycle<N>(S.stack, S.residual, a.pre, a.post);
        __syncthreads();
    }
    for (int i = threadIdx.x; i < Tail<N>::kNodes; i += kTailThreads) a.sol[i] = S.stack.level.sol[i];
}

static bool tail_side(int64_t n) { return n == 17 || n == 9 || n == 5 || n == 3; }

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
        case 17: return launch_tail_n<17>(a, s);
        case 9: return launch_tail_n<9>(a, s);
        case 5: return launch_tail_n<5>(a, s);
        case 3: return launch_tail_n<3>(a, s);
    }
    return fail(PB_ERR_INVALID, "cycle: no tail of side %lld", (long long)n);
}

}  // namespace cycle64
}  // namespace pb

using namespace pb;

// `cycles` V(pre, post) cycles of the FP64 multigrid (core.py:141-193) on a
// hierarchy of sides 2^k + 1, finest first, halving down to 3.  grids: per
// level four pointers, (iterate, scratch of the level's size, right-hand side,
// screen); the finest iterate is updated in place, the coarser iterates and
// right-hand sides are scratch.
extern "C" int pb_vcycles_f64(int64_t levels, const int64_t* sides, void* const* grids, double point_weight,
                              int64_t pre, int64_t post, int64_t cycles, void* workspace, size_t workspace_bytes,
                              void* stream) {
    if (levels < 1 || levels > 16 || !sides || !grids || pre < 0 || post < 0 || cycles < 0)
        return fail(PB_ERR_INVALID, "vcycles: bad args");
    for (int64_t l = 0; l < levels; ++l) {
        if (sides[l] != (l + 1 < levels ? 2 * sides[l + 1] - 1 : 3))
            return fail(PB_ERR_INVALID, "vcycles: sides must halve down to 3");
        for (int k = 0; k < 4; ++k)
            if (!grids[4 * l + k]) return fail(PB_ERR_INVALID, "vcycles: null grid");
    }
    if (!workspace || workspace_bytes < pb_residual_workspace_size(sides[0]) + 256)
        return fail(PB_ERR_WORKSPACE, "vcycles: workspace needs %zu bytes", pb_residual_workspace_size(sides[0]) + 256);
    cudaStream_t s = (cudaStream_t)stream;
    auto sol = [&](int64_t l) { return (double*)grids[4 * l]; };
    auto alt = [&](int64_t l) { return (double*)grids[4 * l + 1]; };
    auto rhs = [&](int64_t l) { return (double*)grids[4 * l + 2]; };
    auto screen = [&](int64_t l) { return (const double*)grids[4 * l + 3]; };
    int64_t top = 0;  // first level of the tail
    while (!cycle64::tail_side(sides[top])) ++top;
    cycle64::TailArgs tail = {};
    for (int64_t l = top; l < levels; ++l) tail.screens[l - top] = screen(l);
    tail.rhs = rhs(top);
    tail.sol = sol(top);
    tail.pw = point_weight;
    tail.pre = (int)pre;
    tail.post = (int)post;
    tail.zero_start = top > 0;
    tail.cycles = top > 0 ? 1 : (int)cycles;
    if (top == 0) return cycle64::launch_tail(sides[0], tail, s);
    double* norm = (double*)workspace;
    void* ws = (char*)workspace + 256;
    for (int64_t c = 0; c < cycles; ++c) {
        for (int64_t l = 0; l < top; ++l) {
            const int64_t n = sides[l];
            if (l > 0) PB_TRY(pb_fill_f64(sol(l), n * n * n, 0.0, stream));
            PB_TRY(pb_relax_f64(sol(l), rhs(l), screen(l), n, point_weight, pre, stream));
            PB_TRY(pb_residual_f64(sol(l), rhs(l), screen(l), alt(l), n, point_weight, norm, ws, workspace_bytes - 256,
                                   stream));
            PB_TRY(pb_restrict_f64(alt(l), rhs(l + 1), n, stream));
        }
        PB_TRY(cycle64::launch_tail(sides[top], tail, s));
        for (int64_t l = top - 1; l >= 0; --l) {
            PB_TRY(pb_prolong_add_f64(sol(l + 1), sol(l), sides[l], stream));
            PB_TRY(pb_relax_f64(sol(l), rhs(l), screen(l), sides[l], point_weight, post, stream));
        }
    }
    return PB_OK;
}
