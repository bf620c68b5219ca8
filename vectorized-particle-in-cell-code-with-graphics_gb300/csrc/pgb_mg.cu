/*
 * Multigrid solver of the Poisson modes FMG_REF (FP64), FMG32 and FP32_DC.
 *
 * Reference path: Mglin (mglin.cpp:21-196): restriction of the right-hand
 * side to every level, the exact 3x3 solve, then for each finer level the
 * interpolation of the coarser solution and two V(1,1) cycles with
 * red-black Gauss-Seidel, half-weighted residuals and bilinear corrections.
 *
 * Compiled with --fmad=false, and every value is the one that the
 * reference's sequence of roundings gives, so that the FP64 form returns
 * the reference's potential bit for bit.  FP64 runs at 1.7 lane-operations
 * per clock and SM here (an addition occupies a scheduler for 64 clocks),
 * so the FP64 forms below do without the operations that round nothing:
 *   - a factor 1/4, 1/2 or 1/8 is a subtraction from the exponent field;
 *   - 4u enters a sum as fma(-4, u, s), 0.5 c + 0.125 t is (4c + t)/8, and
 *     u + 0.5 (a + b) is fma(0.5, a + b, u): the products are exact, so
 *     the one rounding left is the reference's;
 *   - a residual that several coarse points share is computed once;
 *   - a sweep reads only the other colour, so only the black points are
 *     interpolated or corrected before a sweep that starts with red;
 *   - a correction starts at 0, so its first red sweep is (0 - h^2 f)/4.
 *
 * Who works on a level (Cfg):
 *   n <= 17 (FP64), 33 (FP32)   one CTA, every level in shared memory
 *   up to n = 65 (FP64), 129 (FP32)
 *                   a cluster of 16 CTAs in the same launch, a band of rows
 *                   per CTA with the halo that makes one exchange (through
 *                   the CTAs' shared memory, a cluster barrier of 400
 *                   clocks) enough for smoothing, residual and restriction,
 *                   and one for correction and smoothing
 *   above           two launches per level and V-cycle on tiles
 */
#include <cuda_runtime.h>
#include <math.h>
#include "pgb_internal.h"

namespace {

/* ------------------------------------------------------ exact scalings */
/* x * 2^-K for K = 1, 2, 3 */
template <int K>
__device__ __forceinline__ double down_pow2(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    const unsigned a = (unsigned)hi & 0x7fffffffu;
    /* normal before and after: the exponent field drops by K; +-0 stays */
    const bool normal = a - ((unsigned)(K + 1) << 20) < 0x7ff00000u - ((unsigned)(K + 1) << 20);
    const bool zero = (a | (unsigned)lo) == 0u;
    double r = __hiloint2double(normal ? hi - (K << 20) : hi, lo);
    if (!(normal || zero)) r = x * (1.0 / (1 << K));   /* subnormal results, infinities, NaN */
    return r;
}
template <int K>
__device__ __forceinline__ float down_pow2(float x) { return x * (1.0f / (1 << K)); }

__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }

/* the relaxed value from the four neighbours' values (mglin.cpp:116-127) and h^2 f */
template <class T>
__device__ __forceinline__ T gs_value(T ip, T im, T jp, T jm, T g) { return down_pow2<2>(ip + im + jp + jm - g); }
/* minus the residual (mglin.cpp:133-141) */
template <class T>
__device__ __forceinline__ T resid_value(T ip, T im, T jp, T jm, T c, T f, T h2i) {
    return -h2i * fma_t((T)-4, c, ip + im + jp + jm) + f;
}
/* half weighting 0.5 c + 0.125 (ip + im + jp + jm) (mglin.cpp:151-160) */
template <class T>
__device__ __forceinline__ T half_weight(T c, T ip, T im, T jp, T jm) { return down_pow2<3>(fma_t((T)4, c, ip + im + jp + jm)); }

/* the two coarse points whose mean is the bilinear interpolation at a
 * black point (i + j odd: one index even, one odd; mglin.cpp:70-82), in
 * the order in which they are added                                     */
__device__ __forceinline__ void black_pair(int i, int j, int nc, int& k1, int& k0) {
    if (j & 1) {
        k1 = (i >> 1) * nc + ((j + 1) >> 1);
        k0 = (i >> 1) * nc + ((j - 1) >> 1);
    } else {
        k1 = ((i + 1) >> 1) * nc + (j >> 1);
        k0 = ((i - 1) >> 1) * nc + (j >> 1);
    }
}

/* how a V-cycle's first smoothing starts */
enum { FROM_ZERO = 0, FROM_U = 1, FROM_COARSE = 2 };

/* a correction's first red value (0 - g)/4: +0 for g = +-0, else -g/4 */
__device__ __forceinline__ double red_from_zero(double g) {
    const int hi = __double2hiint(g), lo = __double2loint(g);
    const unsigned a = (unsigned)hi & 0x7fffffffu;
    const bool normal = a - (3u << 20) < 0x7ff00000u - (3u << 20), zero = (a | (unsigned)lo) == 0u;
    double r = __hiloint2double(normal ? (hi ^ (int)0x80000000) - (2 << 20) : 0, lo);
    if (!(normal || zero)) r = (0.0 - g) * 0.25;
    return r;
}
__device__ __forceinline__ float red_from_zero(float g) { return (0.0f - g) * 0.25f; }

/* A level's h^2 and 1/h^2, rounded as the reference rounds them, from the
 * host: a division in FP64 is a chain of some ten operations of 64 clocks */
template <class T>
struct MgConst {
    T h2[PGB_MAX_LEVELS], h2i[PGB_MAX_LEVELS];
    T c0;   /* -h * h of the 3x3 grid */
};

/* level l has n_l = 2^(l+1) + 1 nodes a side */
__host__ __device__ constexpr int sm_n(int l) { return (2 << l) + 1; }
__host__ __device__ constexpr int sm_below(int l) { return l == 0 ? 0 : sm_below(l - 1) + sm_n(l - 1) * sm_n(l - 1); }

/* TOP: the finest level that one CTA solves.  FP64: 17 nodes (a level of 33
 * nodes takes 7.3 us in one CTA, bound by its FP64 pipe, and 2.9 us on the
 * cluster); FP32: 33 nodes (1.0 us in one CTA).  CL: the finest that the
 * cluster solves.  FP64: 65 nodes, as 129 keep the FP64 pipes of 16 SMs busy
 * (a visit 15 us, two tile launches 10; the whole solve at 129^2, 257^2 and
 * 513^2 152, 225 and 342 us on the cluster, 139, 204 and 313 in tiles);
 * FP32: 129 (a visit 3.7 us, less than two launches).                    */
template <class T>
struct Cfg;
template <>
struct Cfg<double> { static constexpr int TOP = 3, CL = 5, THREADS = 256; };
template <>
struct Cfg<float> { static constexpr int TOP = 4, CL = 6, THREADS = 512; };

/* ----------------------------------------------------- levels in one CTA */
/* shared image: U, F, G = h^2 F of levels 0..TOP (a V-cycle's top), V, R,
 * GR = h^2 R of levels 0..TOP-1 (below its top), one residual plane      */
template <class T>
struct Sm {
    static constexpr int TOP = Cfg<T>::TOP, A = sm_below(TOP + 1), B = sm_below(TOP);
    static constexpr int WORDS = 3 * A + 3 * B + sm_n(TOP) * sm_n(TOP);
};

extern __shared__ __align__(16) unsigned char mg_smem[];
template <class T>
__device__ __forceinline__ T* smem() { return reinterpret_cast<T*>(mg_smem); }

template <class T, int L, bool TOP>
struct Arr {
    static constexpr int A = Sm<T>::A, B = Sm<T>::B, o = sm_below(L);
    static __device__ __forceinline__ T* u() { return smem<T>() + (TOP ? o : 3 * A + o); }
    static __device__ __forceinline__ T* f() { return smem<T>() + (TOP ? A + o : 3 * A + B + o); }
    static __device__ __forceinline__ T* g() { return smem<T>() + (TOP ? 2 * A + o : 3 * A + 2 * B + o); }
};
template <class T>
__device__ __forceinline__ T* sm_res() { return smem<T>() + 3 * Sm<T>::A + 3 * Sm<T>::B; }

/* who works on a level: one warp for n <= 9, 128 threads for n = 17, 512
 * for n = 33.  Every point is updated by the same arithmetic whichever team
 * updates it.                                                            */
template <int L>
struct Team {
    static constexpr int size = L <= 2 ? 32 : L == 3 ? 128 : 512;
    static __device__ __forceinline__ void sync() {
        if (L <= 2) __syncwarp();
        else if (L == 3) asm volatile("bar.sync 1, 128;" ::: "memory");
        else __syncthreads();
    }
};

/* One V-cycle's work on level L.  A thread keeps its red and its black
 * point (each colour has at most one point per thread) and the shared
 * index arithmetic is done once.                                         */
template <class T, int L, bool TOP, int START>
__device__ __forceinline__ void sm_level_down(const MgConst<T>& c, int kr, int kb, bool hr, bool hb, int b1, int b0) {
    using A = Arr<T, L, TOP>;
    using C = Arr<T, L - 1, false>;
    constexpr int n = sm_n(L), nc = sm_n(L - 1), per = 1 << L, S = Team<L>::size;
    T* const u = A::u();
    const T* const f = A::f();
    const T* const g = A::g();
    const T h2i = c.h2i[L];
    if (START == FROM_COARSE) {
        const T* const uc = Arr<T, L - 1, true>::u();
        if (hb) u[kb] = down_pow2<1>(uc[b1] + uc[b0]);
        Team<L>::sync();
    }
    if (START != FROM_ZERO) {   /* else the red points are there */
        if (hr) u[kr] = gs_value(u[kr + n], u[kr - n], u[kr + 1], u[kr - 1], g[kr]);
        Team<L>::sync();
    }
    if (hb) u[kb] = gs_value(u[kb + n], u[kb - n], u[kb + 1], u[kb - 1], g[kb]);
    Team<L>::sync();
    /* residuals where the restriction reads them: all points of even rows,
     * the black points (even columns) of odd rows                        */
    T* const res = sm_res<T>();
    constexpr int na = (per - 1) * 2 * per, nb = per * per, trips = (na + nb + S - 1) / S;
    T rv[trips];
    int rk[trips];
#pragma unroll
    for (int q = 0; q < trips; ++q) {
        const int t = threadIdx.x + q * S, s = t - na;
        const int i = s < 0 ? 2 * (t >> (L + 1)) + 2 : 2 * (s >> L) + 1;
        const int j = s < 0 ? 1 + (t & (2 * per - 1)) : 2 * (s & (per - 1)) + 2;
        const bool ok = t < na + nb && j <= n - 2;
        const int k = ok ? i * n + j : n + 1;
        rv[q] = resid_value(u[k + n], u[k - n], u[k + 1], u[k - 1], u[k], f[k], h2i);
        rk[q] = ok ? k : -1;
    }
#pragma unroll
    for (int q = 0; q < trips; ++q)
        if (rk[q] >= 0) res[rk[q]] = rv[q];
    Team<L>::sync();
    /* half weighting; the coarse red points get their first value here */
    const T h2c = c.h2[L - 1];
    const int t = threadIdx.x, ic = (t >> L) + 1, jc = 1 + (t & (per - 1));
    if (t < (nc - 2) * per && jc <= nc - 2) {
        const int k = 2 * ic * n + 2 * jc, kc = ic * nc + jc;
        const T r = half_weight(res[k], res[k + n], res[k - n], res[k + 1], res[k - 1]);
        const T gg = h2c * r;
        C::f()[kc] = r;
        C::g()[kc] = gg;
        if (((ic + jc) & 1) == 0) C::u()[kc] = red_from_zero(gg);
    }
    Team<L>::sync();
}
template <class T, int L, bool TOP>
__device__ __forceinline__ void sm_level_up(int kr, int kb, bool hr, bool hb, int b1, int b0) {
    constexpr int n = sm_n(L);
    T* const u = Arr<T, L, TOP>::u();
    const T* const g = Arr<T, L, TOP>::g();
    const T* const vc = Arr<T, L - 1, false>::u();
    if (hb) u[kb] = fma_t((T)0.5, vc[b1] + vc[b0], u[kb]);
    Team<L>::sync();
    if (hr) u[kr] = gs_value(u[kr + n], u[kr - n], u[kr + 1], u[kr - 1], g[kr]);
    Team<L>::sync();
    if (hb) u[kb] = gs_value(u[kb + n], u[kb - n], u[kb + 1], u[kb - 1], g[kb]);
    Team<L>::sync();
}
/* V-cycle with top L; entered by the team of level L */
template <class T, int L, bool TOP, int START>
struct SmV {
    static __device__ __noinline__ void run(const MgConst<T>& mc) {
        constexpr int n = sm_n(L), per = 1 << L;
        static_assert((n - 2) * per <= Team<L>::size, "one point of a colour per thread");
        const int t = threadIdx.x, i = (t >> L) + 1, c = 2 * (t & (per - 1)) + 1;
        const int jr = c + ((i + 1) & 1), jb = c + (i & 1);
        const bool in = i <= n - 2, hr = in && jr <= n - 2, hb = in && jb <= n - 2;
        int b1 = 0, b0 = 0;
        if (hb) black_pair(i, jb, sm_n(L - 1), b1, b0);
        sm_level_down<T, L, TOP, START>(mc, i * n + jr, i * n + jb, hr, hb, b1, b0);
        if (Team<L - 1>::size < Team<L>::size) {
            if (threadIdx.x < Team<L - 1>::size) SmV<T, L - 1, false, FROM_ZERO>::run(mc);
            Team<L>::sync();
        } else {
            SmV<T, L - 1, false, FROM_ZERO>::run(mc);
        }
        sm_level_up<T, L, TOP>(i * n + jr, i * n + jb, hr, hb, b1, b0);
    }
};
/* the 3x3 grid: u = -h^2 f / 4 (mglin.cpp:103-110) */
template <class T, bool TOP, int START>
struct SmV<T, 0, TOP, START> {
    static __device__ __forceinline__ void run(const MgConst<T>& mc) {
        if (threadIdx.x == 0) Arr<T, 0, TOP>::u()[4] = down_pow2<2>(mc.c0 * Arr<T, 0, TOP>::f()[4]);
        Team<0>::sync();
    }
};

/* zero walls of U and V (the other arrays' walls are not read) */
template <class T, int L, bool TOP>
__device__ __forceinline__ void sm_walls(int t) {
    constexpr int n = sm_n(L);
    T* const u = Arr<T, L, TOP>::u();
    if (t >= 0 && t < n) u[t] = u[(n - 1) * n + t] = u[t * n] = u[t * n + n - 1] = (T)0;
    if constexpr (L > 0) sm_walls<T, L - 1, TOP>(t - n);
}
/* F of level L (and G) from get(i, j) of its interior */
template <class T, int L, class Get>
__device__ __forceinline__ void sm_load_f(Get get, const MgConst<T>& mc, bool red) {
    using A = Arr<T, L, true>;
    constexpr int n = sm_n(L), W = 2 << L, trips = (W * W + Cfg<T>::THREADS - 1) / Cfg<T>::THREADS;
    const T h2 = mc.h2[L];
    T v[trips];
#pragma unroll
    for (int q = 0; q < trips; ++q) {
        const int t = threadIdx.x + q * Cfg<T>::THREADS, i = t >> (L + 1), j = t & (W - 1);
        v[q] = (i > 0 && j > 0 && i < W) ? get(i, j) : (T)0;
    }
    sm_walls<T, L, true>(threadIdx.x);
    if constexpr (L > 0) sm_walls<T, L - 1, false>((int)threadIdx.x - Cfg<T>::THREADS / 2);
#pragma unroll
    for (int q = 0; q < trips; ++q) {
        const int t = threadIdx.x + q * Cfg<T>::THREADS, i = t >> (L + 1), j = t & (W - 1);
        if (i > 0 && j > 0 && i < W) {
            const T g = h2 * v[q];
            A::f()[i * n + j] = v[q];
            A::g()[i * n + j] = g;
            if (red && ((i + j) & 1) == 0) A::u()[i * n + j] = red_from_zero(g);
        }
    }
    __syncthreads();
}
template <class T, int L>
__device__ __forceinline__ void sm_store_u(T* gu) {
    constexpr int n = sm_n(L), W = 2 << L;
#pragma unroll
    for (int t = threadIdx.x; t < W * W; t += Cfg<T>::THREADS) {
        const int i = t >> (L + 1), j = t & (W - 1);
        if (i > 0 && j > 0) gu[i * n + j] = Arr<T, L, true>::u()[i * n + j];
    }
    __syncthreads();
}
/* F of level L from F of level L+1 (interior) */
template <class T, int L>
__device__ __forceinline__ void sm_restrict_f(const MgConst<T>& mc) {
    using A = Arr<T, L, true>;
    constexpr int n = sm_n(L), nf = sm_n(L + 1), W = 2 << L;
    const T h2 = mc.h2[L];
    const T* const ff = Arr<T, L + 1, true>::f();
    for (int t = threadIdx.x; t < W * W; t += Cfg<T>::THREADS) {
        const int i = t >> (L + 1), j = t & (W - 1);
        if (i > 0 && j > 0) {
            const int q = 2 * i * nf + 2 * j;
            const T f = half_weight(ff[q], ff[q + nf], ff[q - nf], ff[q + 1], ff[q - 1]);
            A::f()[i * n + j] = f;
            A::g()[i * n + j] = h2 * f;
        }
    }
    __syncthreads();
}
/* F of the levels below L, then the full multigrid up to level L */
template <class T, int L>
struct SmF {
    static __device__ __forceinline__ void restrict_all(const MgConst<T>& mc) {
        sm_restrict_f<T, L - 1>(mc);
        SmF<T, L - 1>::restrict_all(mc);
    }
    static __device__ __forceinline__ void solve(const MgConst<T>& mc) {
        SmF<T, L - 1>::solve(mc);
        __syncthreads();
        if (threadIdx.x < Team<L>::size) {
            SmV<T, L, true, FROM_COARSE>::run(mc);
            SmV<T, L, true, FROM_U>::run(mc);
        }
    }
};
template <class T>
struct SmF<T, 0> {
    static __device__ __forceinline__ void restrict_all(const MgConst<T>&) {}
    static __device__ __forceinline__ void solve(const MgConst<T>& mc) {
        if (threadIdx.x < Team<0>::size) SmV<T, 0, true, FROM_U>::run(mc);
    }
};
/* full multigrid at level L, right-hand side f (one CTA) */
template <class T, int L>
__device__ __forceinline__ void sm_fmg(const T* f, const MgConst<T>& mc) {
    sm_load_f<T, L>([f](int i, int j) { return __ldcg(f + i * sm_n(L) + j); }, mc, false);
    SmF<T, L>::restrict_all(mc);
    SmF<T, L>::solve(mc);
    __syncthreads();
}
/* one V-cycle from 0 at level L, right-hand side f (one CTA) */
template <class T, int L>
__device__ __forceinline__ void sm_vcycle0(const T* f, const MgConst<T>& mc) {
    sm_load_f<T, L>([f](int i, int j) { return __ldcg(f + i * sm_n(L) + j); }, mc, true);
    if (threadIdx.x < Team<L>::size) SmV<T, L, true, FROM_ZERO>::run(mc);
    __syncthreads();
}

/* ------------------------------------------------------------- tiles */
/* M x N coarse points (from row ic0, column jc0) and their 2M x 2N fine
 * points (rows 2 ic0 - 1 ...): a tile loads the halo that lets it do
 * everything between two exchanges by itself.  The halo's values are
 * computed by the neighbouring tiles too, from the same inputs, so they
 * agree.  Loads go past L1 (__ldcg): in a cluster, other CTAs wrote the
 * data in this launch.                                                  */
template <int M, int N>
struct Tile {
    static constexpr int UR = 2 * M + 7, UC = 2 * N + 7;   /* u: rows 2 ic0 - 4 ... */
    static constexpr int FR = 2 * M + 5, FC = 2 * N + 5;   /* f: rows 2 ic0 - 3 ... */
    static constexpr int RR = 2 * M + 1, RC = 2 * N + 1;   /* residual: rows 2 ic0 - 1 ... */
    static constexpr int WORDS = UR * UC + FR * FC + RR * RC;
};

/* first smoothing (from u, from the interpolated coarse solution uc, or
 * from 0) of the tile into w, and the half-weighted residual into rc    */
template <class T, int M, int N, int START, int THREADS>
__device__ __forceinline__ void tile_down(const T* u, const T* uc, const T* f, T* w, T* rc, int n, int ic0, int jc0,
                                          T h2, T h2i) {
    using L = Tile<M, N>;
    T* const su = reinterpret_cast<T*>(mg_smem);
    T* const sf = su + L::UR * L::UC;
    T* const sr = sf + L::FR * L::FC;
    const int nc = n / 2 + 1;
    const int iu = 2 * ic0 - 4, ju = 2 * jc0 - 4;
    /* black points from their source; walls 0; red points are written below */
#pragma unroll 2
    for (int t = threadIdx.x; t < L::UR * L::UC; t += THREADS) {
        const int a = t / L::UC, b = t - a * L::UC, i = iu + a, j = ju + b;
        T v = (T)0;
        if (START != FROM_ZERO && i > 0 && j > 0 && i < n - 1 && j < n - 1) {
            if (START == FROM_U) v = __ldcg(u + i * n + j);
            else if ((i + j) & 1) {
                int k1, k0;
                black_pair(i, j, nc, k1, k0);
                v = down_pow2<1>(__ldcg(uc + k1) + __ldcg(uc + k0));
            }
        }
        su[t] = v;
    }
#pragma unroll 2
    for (int t = threadIdx.x; t < L::FR * L::FC; t += THREADS) {
        const int a = t / L::FC, b = t - a * L::FC, i = iu + 1 + a, j = ju + 1 + b;
        sf[t] = (i > 0 && j > 0 && i < n - 1 && j < n - 1) ? __ldcg(f + i * n + j) : (T)0;
    }
    __syncthreads();
    /* red on the whole f region, black one point further in */
#pragma unroll
    for (int color = 0; color < 2; ++color) {
        const int rows = L::FR - 2 * color, slots = N + 3 - color;
        for (int t = threadIdx.x; t < rows * slots; t += THREADS) {
            const int a = t / slots, i = iu + 1 + color + a;
            /* first column of the region with the colour's parity */
            const int jf = ju + 1 + color;
            const int j = jf + ((i + jf + color) & 1) + 2 * (t - a * slots);
            if (i > 0 && j > 0 && i < n - 1 && j < n - 1 && j <= ju + L::FC - color) {
                const int k = (i - iu) * L::UC + (j - ju);
                const T g = h2 * sf[(i - iu - 1) * L::FC + (j - ju - 1)];
                if (START == FROM_ZERO && color == 0) su[k] = red_from_zero(g);
                else su[k] = gs_value(su[k + L::UC], su[k - L::UC], su[k + 1], su[k - 1], g);
            }
        }
        __syncthreads();
    }
    /* residuals on even rows, and at even columns of odd rows */
    for (int t = threadIdx.x; t < M * L::RC + (M + 1) * N; t += THREADS) {
        const int s = t - M * L::RC;
        int a, b;   /* row and column of the residual region */
        if (s < 0) {
            const int q = t / L::RC;
            a = 2 * q + 1;
            b = t - q * L::RC;
        } else {
            const int q = s / N;
            a = 2 * q;
            b = 2 * (s - q * N) + 1;
        }
        const int i = iu + 3 + a, j = ju + 3 + b;
        if (i < n - 1 && j < n - 1) {
            const int k = (a + 3) * L::UC + b + 3;
            sr[a * L::RC + b] = resid_value(su[k + L::UC], su[k - L::UC], su[k + 1], su[k - 1], su[k],
                                            sf[(a + 2) * L::FC + b + 2], h2i);
        }
    }
    /* the tile's own smoothed points */
    for (int t = threadIdx.x; t < 4 * M * N; t += THREADS) {
        const int a = t / (2 * N), b = t - a * (2 * N), i = iu + 3 + a, j = ju + 3 + b;
        if (i < n - 1 && j < n - 1) w[i * n + j] = su[(a + 3) * L::UC + b + 3];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < M * N; t += THREADS) {
        const int a = t / N, b = t - a * N, ic = ic0 + a, jc = jc0 + b;
        if (ic < nc - 1 && jc < nc - 1) {
            const T* const r = sr + (2 * a + 1) * L::RC + 2 * b + 1;
            rc[ic * nc + jc] = half_weight(r[0], r[L::RC], r[-L::RC], r[1], r[-1]);
        }
    }
    __syncthreads();   /* the tile's shared memory may be used again */
}

/* w plus the coarse correction vc, smoothed, into u */
template <class T, int M, int N, int THREADS>
__device__ __forceinline__ void tile_up(const T* w, const T* vc, const T* f, T* u, int n, int ic0, int jc0, T h2) {
    constexpr int UR = 2 * M + 4, UC = 2 * N + 4, FR = 2 * M + 2, FC = 2 * N + 2;
    T* const su = reinterpret_cast<T*>(mg_smem);
    T* const sf = su + UR * UC;
    const int nc = n / 2 + 1;
    const int iu = 2 * ic0 - 3, ju = 2 * jc0 - 3;
#pragma unroll 2
    for (int t = threadIdx.x; t < UR * UC; t += THREADS) {
        const int a = t / UC, b = t - a * UC, i = iu + a, j = ju + b;
        T v = (T)0;
        if (((i + j) & 1) && i > 0 && j > 0 && i < n - 1 && j < n - 1) {
            int k1, k0;
            black_pair(i, j, nc, k1, k0);
            v = fma_t((T)0.5, __ldcg(vc + k1) + __ldcg(vc + k0), __ldcg(w + i * n + j));
        }
        su[t] = v;
    }
#pragma unroll 2
    for (int t = threadIdx.x; t < FR * FC; t += THREADS) {
        const int a = t / FC, b = t - a * FC, i = iu + 1 + a, j = ju + 1 + b;
        sf[t] = (i > 0 && j > 0 && i < n - 1 && j < n - 1) ? h2 * __ldcg(f + i * n + j) : (T)0;
    }
    __syncthreads();
#pragma unroll
    for (int color = 0; color < 2; ++color) {
        const int rows = FR - 2 * color, slots = N + 1 - color;
        for (int t = threadIdx.x; t < rows * slots; t += THREADS) {
            const int a = t / slots, i = iu + 1 + color + a;
            const int jf = ju + 1 + color;
            const int j = jf + ((i + jf + color) & 1) + 2 * (t - a * slots);
            if (i > 0 && j > 0 && i < n - 1 && j < n - 1) {
                const int k = (i - iu) * UC + (j - ju);
                su[k] = gs_value(su[k + UC], su[k - UC], su[k + 1], su[k - 1], sf[(i - iu - 1) * FC + (j - ju - 1)]);
            }
        }
        __syncthreads();
    }
    for (int t = threadIdx.x; t < 4 * M * N; t += THREADS) {
        const int a = t / (2 * N), b = t - a * (2 * N), i = iu + 2 + a, j = ju + 2 + b;
        if (i < n - 1 && j < n - 1) u[i * n + j] = su[(a + 2) * UC + b + 2];
    }
    __syncthreads();
}

/* ------------------------------------------ levels on the whole GPU */
#define MG_THREADS 256
template <class T, int M, int N, int START>
__global__ void __launch_bounds__(MG_THREADS) k_mg_down(const T* u, const T* uc, const T* f, T* w, T* rc, int n, T h2,
                                                        T h2i) {
    pgb_pdl_entry();
    tile_down<T, M, N, START, MG_THREADS>(u, uc, f, w, rc, n, 1 + M * blockIdx.y, 1 + N * blockIdx.x, h2, h2i);
}
template <class T, int M, int N>
__global__ void __launch_bounds__(MG_THREADS) k_mg_up(const T* w, const T* vc, const T* f, T* u, int n, T h2) {
    pgb_pdl_entry();
    tile_up<T, M, N, MG_THREADS>(w, vc, f, u, n, 1 + M * blockIdx.y, 1 + N * blockIdx.x, h2);
}
/* right-hand side of the coarser level (interior) */
template <class T>
__global__ void k_mg_restrict(T* fc, const T* ff, int nc) {
    pgb_pdl_entry();
    const int nf = 2 * nc - 1;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nc * nc; k += gridDim.x * blockDim.x) {
        const int i = k / nc, j = k - i * nc;
        if (i > 0 && j > 0 && i < nc - 1 && j < nc - 1) {
            const T* const q = ff + 2 * i * nf + 2 * j;
            fc[k] = half_weight(q[0], q[nf], q[-nf], q[1], q[-1]);
        }
    }
}

/* ------------------------------------------- levels in one launch */
constexpr int CL_CTAS = 16;
/* level arrays in global memory */
template <class T>
struct MgPtrs {
    T* u[PGB_MAX_LEVELS];
    T* f[PGB_MAX_LEVELS];
    T* v[PGB_MAX_LEVELS];
    T* r[PGB_MAX_LEVELS];
    T* w[PGB_MAX_LEVELS];
    MgConst<T> c;
};

/* every CTA's writes before are seen by every CTA's reads after */
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ int cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
/* *p as CTA `rank` of the cluster holds it in its shared memory */
__device__ __forceinline__ unsigned remote_addr(const void* p, int rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ double remote(const double* p, int rank) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(remote_addr(p, rank)));
    return v;
}
__device__ __forceinline__ float remote(const float* p, int rank) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote_addr(p, rank)));
    return v;
}

/* The band of a CTA on level L: coarse rows ic0 = 1 + M rank ... and their
 * fine rows 2 ic0 - 1 ..., whole rows, with the halo that makes the
 * smoothing, the residual, the restriction and, later, the correction and
 * its smoothing local.  Between the levels, and from one V-cycle to the
 * next, a CTA reads the rows it needs from the shared memory of the CTAs
 * that own them: a cluster barrier costs 400 clocks when only shared memory
 * was written before it, 2000 when global stores were.                   */
template <class T, int L>
struct Band {
    static constexpr int n = sm_n(L), N = 1 << L, M = N / CL_CTAS;
    static constexpr int UR = 2 * M + 8;   /* u: rows 2 ic0 - 5 ...       */
    static constexpr int GR = 2 * M + 6;   /* g: rows 2 ic0 - 4 ...       */
    static constexpr int FR = 2 * M + 1;   /* f, residual: rows 2 ic0 - 1 ... */
    static constexpr int WORDS = (UR + GR + 2 * FR) * n + M * sm_n(L - 1);
    static constexpr int BASE = Sm<T>::WORDS + [] {
        if constexpr (L > Cfg<T>::TOP + 1) return Band<T, L - 1>::END;
        else return 0;
    }();
    static constexpr int END = BASE - Sm<T>::WORDS + WORDS;
    static __device__ __forceinline__ T* u() { return smem<T>() + BASE; }
    static __device__ __forceinline__ T* g() { return u() + UR * n; }
    static __device__ __forceinline__ T* f() { return g() + GR * n; }
    static __device__ __forceinline__ T* res() { return f() + FR * n; }
    static __device__ __forceinline__ T* rc() { return res() + FR * n; }   /* restricted residual: coarse rows ic0 ... */
    /* u at fine row i (not a wall) from its owner */
    static __device__ __forceinline__ T owner_u(int i, int j) {
        const int o = (i - 1) / (2 * M);
        return remote(u() + (i - 2 * M * o + 3) * n + j, o);
    }
    /* the restricted residual at coarse row i (interior) from its owner */
    static __device__ __forceinline__ T owner_rc(int i, int j) {
        const int o = (i - 1) / M;
        return remote(rc() + (i - 1 - M * o) * sm_n(L - 1) + j, o);
    }
};
/* u of level L at row i (any), column j: from the level's bands, or from the
 * first CTA                                                              */
template <class T, int L>
__device__ __forceinline__ T cluster_u(int i, int j) {
    if constexpr (L > Cfg<T>::TOP) return i > 0 && i < sm_n(L) - 1 ? Band<T, L>::owner_u(i, j) : (T)0;
    else return remote(Arr<T, L, true>::u() + i * sm_n(L) + j, 0);
}
/* the sum of the two coarse values whose mean is the interpolation at black
 * point (i, j) of level L (black_pair)                                   */
template <class T, int L>
__device__ __forceinline__ T coarse_pair(int i, int j) {
    if (j & 1) return cluster_u<T, L - 1>(i >> 1, (j + 1) >> 1) + cluster_u<T, L - 1>(i >> 1, (j - 1) >> 1);
    return cluster_u<T, L - 1>((i + 1) >> 1, j >> 1) + cluster_u<T, L - 1>((i - 1) >> 1, j >> 1);
}
/* one colour on `rows` band rows from row i0: a row has N slots */
template <class T, int L>
__device__ __forceinline__ void band_sweep(int color, int i0, int rows, int iu) {
    using B = Band<T, L>;
    constexpr int n = B::n;
    T* const u = B::u();
    const T* const g = B::g();
#pragma unroll 2
    for (int t = threadIdx.x; t < rows << L; t += Cfg<T>::THREADS) {
        const int i = i0 + (t >> L), j = 1 + ((i + 1 + color) & 1) + 2 * (t & (B::N - 1));
        if (i > 0 && i < n - 1 && j < n - 1) {
            const int k = (i - iu) * n + j;
            u[k] = gs_value(u[k + n], u[k - n], u[k + 1], u[k - 1], g[k - n]);
        }
    }
    __syncthreads();
}
template <class T, int L, int START, bool ABOVE>
__device__ __forceinline__ void cl_vcycle(const MgPtrs<T>& p, const T* gf);
/* one V-cycle from 0 at level L on the residual restricted from level L+1
 * (ABOVE) or on r[L]                                                     */
template <class T, int L, bool ABOVE>
struct ClLower {
    static __device__ __forceinline__ void run(const MgPtrs<T>& p) {
        if constexpr (L > Cfg<T>::TOP) {
            cl_vcycle<T, L, FROM_ZERO, ABOVE>(p, p.r[L]);
        } else {
            if (cluster_rank() == 0) {
                sm_load_f<T, L>([](int i, int j) { return Band<T, L + 1>::owner_rc(i, j); }, p.c, true);
                if (threadIdx.x < Team<L>::size) SmV<T, L, true, FROM_ZERO>::run(p.c);
                __syncthreads();
            }
            cluster_sync();
        }
    }
};
/* V-cycle of level L.  ABOVE: the right-hand side is what level L+1
 * restricted; else it is gf (global), read on the first of two V-cycles and
 * kept for the second (FROM_U).  The result stays in the bands.          */
template <class T, int L, int START, bool ABOVE>
__device__ __forceinline__ void cl_vcycle(const MgPtrs<T>& p, const T* gf) {
    using B = Band<T, L>;
    constexpr int n = B::n, N = B::N, M = B::M, nc = sm_n(L - 1), TH = Cfg<T>::THREADS;
    const int ic0 = 1 + M * cluster_rank(), iu = 2 * ic0 - 5;
    const T h2 = p.c.h2[L], h2i = p.c.h2i[L];
    T* const su = B::u();
    T* const sg = B::g();
    T* const sf = B::f();
    T* const sr = B::res();
    if constexpr (START == FROM_U) {
        /* the halo's black points from their owners; the others are here */
        constexpr int halo = B::UR - 2 * M;
#pragma unroll
        for (int t = threadIdx.x; t < halo << L; t += TH) {
            const int h = t >> L, a = h < 4 ? h : h + 2 * M, i = iu + a, j = 1 + (i & 1) + 2 * (t & (N - 1));
            if (i > 0 && i < n - 1 && j < n - 1) su[a * n + j] = B::owner_u(i, j);
        }
    } else {
        /* the walls, then the black points from their source (a correction: 0) */
        for (int t = threadIdx.x; t < B::UR; t += TH) su[t * n] = su[t * n + n - 1] = (T)0;
#pragma unroll 4
        for (int t = threadIdx.x; t < B::UR << L; t += TH) {
            const int a = t >> L, i = iu + a, c = 2 * (t & (N - 1)) + 1, j = c + (i & 1);
            T v = (T)0;
            if (START == FROM_COARSE && i > 0 && i < n - 1 && j < n - 1) v = down_pow2<1>(coarse_pair<T, L>(i, j));
            if (j < n - 1) su[a * n + j] = v;
            /* a wall row's red points are read as 0 too */
            const int jr = c + ((i + 1) & 1);
            if ((i <= 0 || i >= n - 1) && jr < n - 1) su[a * n + jr] = (T)0;
        }
        /* g on the red region, f where residuals are taken; a correction's
         * red points start from g                                        */
#pragma unroll 4
        for (int t = threadIdx.x; t < B::GR << (L + 1); t += TH) {
            const int a = t >> (L + 1), j = t & (2 * N - 1), i = iu + 1 + a;
            if (i > 0 && i < n - 1 && j > 0) {
                T v;
                if constexpr (ABOVE) v = Band<T, L + 1>::owner_rc(i, j);
                else v = __ldcg(gf + i * n + j);
                const T g = h2 * v;
                sg[a * n + j] = g;
                const int b = a - 3;
                if (b >= 0 && b < B::FR) sf[b * n + j] = v;
                if (START == FROM_ZERO && ((i + j) & 1) == 0) su[(a + 1) * n + j] = red_from_zero(g);
            }
        }
    }
    /* a neighbour may still be reading this band's black points (FROM_U):
     * they change in the black sweep                                     */
    if (START == FROM_U) cluster_arrive();
    __syncthreads();
    if (START != FROM_ZERO) band_sweep<T, L>(0, iu + 1, B::GR, iu);
    if (START == FROM_U) cluster_wait();
    band_sweep<T, L>(1, iu + 2, B::GR - 2, iu);
    /* residuals: even rows 2 ic0 ... whole, odd rows at even columns */
#pragma unroll 2
    for (int t = threadIdx.x; t < (M << (L + 1)) + ((M + 1) << L); t += TH) {
        const int s = t - (M << (L + 1));
        const int b = s < 0 ? 2 * (t >> (L + 1)) + 1 : 2 * (s >> L);
        const int j = s < 0 ? t & (2 * N - 1) : 2 * (s & (N - 1));
        const int i = iu + 4 + b;
        if (j > 0 && i < n - 1) {
            const int k = (b + 4) * n + j;
            sr[b * n + j] = resid_value(su[k + n], su[k - n], su[k + 1], su[k - 1], su[k], sf[b * n + j], h2i);
        }
    }
    __syncthreads();
    T* const rc = B::rc();
    for (int t = threadIdx.x; t < M << L; t += TH) {
        const int a = t >> L, jc = t & (N - 1), ic = ic0 + a;
        if (jc > 0 && ic < nc - 1) {
            const T* const r = sr + (2 * a + 1) * n + 2 * jc;
            rc[a * nc + jc] = half_weight(r[0], r[n], r[-n], r[1], r[-1]);
        }
    }
    cluster_sync();
    ClLower<T, L - 1, true>::run(p);
    /* the correction of the black points, then a sweep */
#pragma unroll 4
    for (int t = threadIdx.x; t < (2 * M + 4) << L; t += TH) {
        const int a = t >> L, i = iu + 2 + a, j = 1 + (i & 1) + 2 * (t & (N - 1));
        if (i > 0 && i < n - 1 && j < n - 1) {
            T& x = su[(a + 2) * n + j];
            x = fma_t((T)0.5, coarse_pair<T, L>(i, j), x);
        }
    }
    __syncthreads();
    band_sweep<T, L>(0, iu + 3, 2 * M + 2, iu);
    band_sweep<T, L>(1, iu + 4, 2 * M, iu);
    cluster_sync();
}
/* the bands' own rows to global memory */
template <class T, int L>
__device__ __forceinline__ void cl_store(T* gu) {
    using B = Band<T, L>;
    const int i0 = 2 * B::M * cluster_rank() + 1;   /* band row 4 */
    for (int t = threadIdx.x; t < (2 * B::M) << (L + 1); t += Cfg<T>::THREADS) {
        const int a = t >> (L + 1), j = t & (2 * B::N - 1), i = i0 + a;
        if (j > 0 && i < B::n - 1) gu[i * B::n + j] = B::u()[(a + 4) * B::n + j];
    }
}
/* right-hand side of level L from level L+1, shared out */
template <class T, int L>
__device__ __forceinline__ void cl_restrict(const MgPtrs<T>& p) {
    constexpr int n = sm_n(L), nf = sm_n(L + 1), W = 2 << L, TH = Cfg<T>::THREADS;
    for (int t = threadIdx.x + TH * cluster_rank(); t < W * W; t += TH * CL_CTAS) {
        const int i = t >> (L + 1), j = t & (W - 1);
        if (i > 0 && j > 0) {
            const T* const q = p.f[L + 1] + 2 * i * nf + 2 * j;
            p.f[L][i * n + j] = half_weight(__ldcg(q), __ldcg(q + nf), __ldcg(q - nf), __ldcg(q + 1), __ldcg(q - 1));
        }
    }
    cluster_sync();
}
template <class T, int L>
struct ClF {
    static __device__ __forceinline__ void run(const MgPtrs<T>& p) {
        if constexpr (L > Cfg<T>::TOP) {
            cl_restrict<T, L - 1>(p);
            ClF<T, L - 1>::run(p);
            cl_vcycle<T, L, FROM_COARSE, false>(p, p.f[L]);
            cl_vcycle<T, L, FROM_U, false>(p, p.f[L]);
        } else {
            if (cluster_rank() == 0) {
                sm_fmg<T, L>(p.f[L], p.c);
                __syncthreads();
            }
            cluster_sync();
        }
    }
};

/* FMG: full multigrid at level J from f[J] into u[J]; else one V-cycle
 * from 0 at level J on the right-hand side r[J] into v[J].  A cluster of
 * CL_CTAS CTAs for J > TOP, one CTA otherwise.                           */
template <class T, int J, bool FMG>
__global__ void __launch_bounds__(Cfg<T>::THREADS) k_mg_levels(const __grid_constant__ MgPtrs<T> p) {
    pgb_pdl_entry();
    if constexpr (J > Cfg<T>::TOP) {
        if constexpr (FMG) ClF<T, J>::run(p);
        else ClLower<T, J, false>::run(p);
        cl_store<T, J>(FMG ? p.u[J] : p.v[J]);
    } else {
        if constexpr (FMG) sm_fmg<T, J>(p.f[J], p.c);
        else sm_vcycle0<T, J>(p.r[J], p.c);
        sm_store_u<T, J>(FMG ? p.u[J] : p.v[J]);
    }
}

/* ====================================================== host side */
template <class T, int J>
constexpr size_t levels_smem() {
    if constexpr (J > Cfg<T>::TOP) return sizeof(T) * (Sm<T>::WORDS + Band<T, J>::END);
    else return sizeof(T) * Sm<T>::WORDS;
}
template <class T, int M, int N>
constexpr size_t tile_smem() { return sizeof(T) * Tile<M, N>::WORDS; }

template <class T>
MgConst<T> mg_const(const pgb_run* r) {
    MgConst<T> c = {};
    const T length = (T)r->p.xlength;
    for (int l = 0; l < r->ng; ++l) {
        const T h = length / (T)(r->mg_n[l] - 1);
        c.h2[l] = h * h;
        c.h2i[l] = (T)1.0 / (h * h);
    }
    const T h0 = (T)0.5 * length;
    c.c0 = -h0 * h0;
    return c;
}
template <class T>
MgPtrs<T> mg_ptrs(pgb_run* r);
template <>
MgPtrs<double> mg_ptrs<double>(pgb_run* r) {
    MgPtrs<double> p;
    for (int l = 0; l < PGB_MAX_LEVELS; ++l) {
        p.u[l] = r->mg_u[l]; p.f[l] = r->mg_f[l]; p.v[l] = r->mg_v[l]; p.r[l] = r->mg_r[l]; p.w[l] = r->mg_w[l];
    }
    p.c = mg_const<double>(r);
    return p;
}
template <>
MgPtrs<float> mg_ptrs<float>(pgb_run* r) {
    MgPtrs<float> p;
    for (int l = 0; l < PGB_MAX_LEVELS; ++l) {
        p.u[l] = r->mg32_u[l]; p.f[l] = r->mg32_f[l]; p.v[l] = r->mg32_v[l]; p.r[l] = r->mg32_r[l]; p.w[l] = r->mg32_w[l];
    }
    p.c = mg_const<float>(r);
    return p;
}

template <class T, int J, bool FMG>
cudaError_t levels_attr() {
    cudaError_t e = cudaFuncSetAttribute(k_mg_levels<T, J, FMG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)levels_smem<T, J>());
    if (e == cudaSuccess && J > Cfg<T>::TOP)
        e = cudaFuncSetAttribute(k_mg_levels<T, J, FMG>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}
template <class T, int J, bool FMG>
int levels_go(pgb_run* r) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(J > Cfg<T>::TOP ? CL_CTAS : 1);
    cfg.blockDim = dim3(Cfg<T>::THREADS);
    cfg.dynamicSmemBytes = levels_smem<T, J>();
    cfg.stream = r->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CL_CTAS;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = J > Cfg<T>::TOP ? 2 : 1;
    PGB_CK(r, cudaLaunchKernelEx(&cfg, k_mg_levels<T, J, FMG>, mg_ptrs<T>(r)));
    r->launches++;
    return 0;
}
template <class T, bool FMG>
int levels_launch(pgb_run* r, int J) {
    switch (J) {
        case 1: return levels_go<T, 1, FMG>(r);
        case 2: return levels_go<T, 2, FMG>(r);
        case 3: return levels_go<T, 3, FMG>(r);
        case 4: return levels_go<T, 4, FMG>(r);
        case 5: return levels_go<T, 5, FMG>(r);
    }
    return levels_go<T, Cfg<T>::CL, FMG>(r);
}
template <class T>
int mg_attrs(pgb_run* r) {
    PGB_CK(r, (levels_attr<T, 1, true>()));
    PGB_CK(r, (levels_attr<T, 2, true>()));
    PGB_CK(r, (levels_attr<T, 3, true>()));
    PGB_CK(r, (levels_attr<T, 4, true>()));
    PGB_CK(r, (levels_attr<T, 5, true>()));
    PGB_CK(r, (levels_attr<T, Cfg<T>::CL, true>()));
    PGB_CK(r, (levels_attr<T, 1, false>()));
    PGB_CK(r, (levels_attr<T, 2, false>()));
    PGB_CK(r, (levels_attr<T, 3, false>()));
    PGB_CK(r, (levels_attr<T, 4, false>()));
    PGB_CK(r, (levels_attr<T, 5, false>()));
    PGB_CK(r, (levels_attr<T, Cfg<T>::CL, false>()));
    return 0;
}
static_assert(tile_smem<double, 8, 8>() <= 48 * 1024, "the tile kernels use no more than the default shared memory");

/* V-cycle at level j > CL (mglin.cpp:176-196): u -> w -> u.  A level has
 * one V-cycle in flight at a time, so one spare buffer w serves.         */
template <class T, int START>
int vcycle(pgb_run* r, const MgPtrs<T>& p, int j, T* u, const T* f, const T* uc);
template <class T, int M, int N, int START>
int vcycle_tiles(pgb_run* r, const MgPtrs<T>& p, int j, T* u, const T* f, const T* uc) {
    const int n = r->mg_n[j], nc = r->mg_n[j - 1];
    const dim3 grid((nc - 2 + N - 1) / N, (nc - 2 + M - 1) / M);
    PGB_CK(r, pgb_launch_pdl(k_mg_down<T, M, N, START>, grid, dim3(MG_THREADS), tile_smem<T, M, N>(), r->stream, (const T*)u,
                             uc, f, p.w[j], p.r[j - 1], n, p.c.h2[j], p.c.h2i[j]));
    r->launches++;
    if (j - 1 > Cfg<T>::CL) {
        if (vcycle<T, FROM_ZERO>(r, p, j - 1, p.v[j - 1], p.r[j - 1], nullptr)) return PGB_ERR_CUDA;
    } else if (levels_launch<T, false>(r, j - 1)) {
        return PGB_ERR_CUDA;
    }
    PGB_CK(r, pgb_launch_pdl(k_mg_up<T, M, N>, grid, dim3(MG_THREADS), tile_smem<T, M, N>(), r->stream, (const T*)p.w[j],
                             (const T*)p.v[j - 1], f, u, n, p.c.h2[j]));
    r->launches++;
    return 0;
}
/* Tiles of 8 x 8 coarse points, 256 of them at 257^2: with 8 x 16, half as
 * many, a block was alone on its SM with its load latencies and barriers
 * (FMG_REF / ten passes of FP32_DC at 257^2 206.6 / 291.8 us, with 8 x 8
 * 203.1 / 278.2; at 513^2 317.7 / 445.9 and 312.0 / 425.7).  4 x 8 at 129
 * nodes (FP64 only), where 8 x 8 are 64 tiles (142.6 and 139.9 us).      */
template <class T, int START>
int vcycle(pgb_run* r, const MgPtrs<T>& p, int j, T* u, const T* f, const T* uc) {
    if constexpr (Cfg<T>::CL < 6)
        if (j == 6) return vcycle_tiles<T, 4, 8, START>(r, p, j, u, f, uc);
    return vcycle_tiles<T, 8, 8, START>(r, p, j, u, f, uc);
}

template <class T>
int fmg(pgb_run* r) {
    constexpr int CL = Cfg<T>::CL;
    const int ng = r->ng;
    const MgPtrs<T> p = mg_ptrs<T>(r);
    for (int j = ng - 2; j >= CL; --j) {
        const int nc = r->mg_n[j], blocks = (nc * nc + 255) / 256;
        PGB_CK(r, pgb_launch_pdl(k_mg_restrict<T>, dim3(blocks), dim3(256), 0, r->stream, p.f[j], (const T*)p.f[j + 1], nc));
        r->launches++;
    }
    if (levels_launch<T, true>(r, ng - 1 < CL ? ng - 1 : CL)) return PGB_ERR_CUDA;
    for (int j = CL + 1; j < ng; ++j) {
        if (vcycle<T, FROM_COARSE>(r, p, j, p.u[j], p.f[j], p.u[j - 1])) return PGB_ERR_CUDA;
        if (vcycle<T, FROM_U>(r, p, j, p.u[j], p.f[j], nullptr)) return PGB_ERR_CUDA;
    }
    PGB_CK(r, cudaGetLastError());
    return 0;
}

}  // namespace

int pgb_mg_attributes(pgb_run* r) { return mg_attrs<double>(r) || mg_attrs<float>(r) ? PGB_ERR_CUDA : 0; }
int pgb_mg_fmg64(pgb_run* r) { return fmg<double>(r); }
int pgb_mg_fmg32(pgb_run* r) { return fmg<float>(r); }
int pgb_mg_vcycle32(pgb_run* r) {
    const MgPtrs<float> p = mg_ptrs<float>(r);
    const int top = r->ng - 1;
    const int rc = top > Cfg<float>::CL ? vcycle<float, FROM_ZERO>(r, p, top, p.v[top], p.r[top], nullptr)
                                : levels_launch<float, false>(r, top);
    if (rc) return rc;
    PGB_CK(r, cudaGetLastError());
    return 0;
}
