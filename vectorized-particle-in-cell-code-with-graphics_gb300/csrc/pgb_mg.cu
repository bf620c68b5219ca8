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
 * Who works on a level:
 *   n <= 33         one CTA, every level in shared memory; n <= 17 on 128
 *                   threads (one warp per scheduler, barrier of 21 clocks)
 *   n = 65, 129     a cluster of 16 CTAs in the same launch, a band of rows
 *                   per CTA with the halo that makes one exchange (through
 *                   L2, a cluster barrier of 380 clocks) enough for
 *                   smoothing, residual and restriction, and one for
 *                   correction and smoothing
 *   n >= 257        two launches per level and V-cycle (the same two tile
 *                   functions on 16 x 32 tiles)
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
    /* normal before and after: the exponent field drops by K */
    if (a - ((unsigned)(K + 1) << 20) < 0x7ff00000u - ((unsigned)(K + 1) << 20)) return __hiloint2double(hi - (K << 20), lo);
    if ((a | (unsigned)lo) == 0u) return x;
    return x * (1.0 / (1 << K));   /* subnormal results, infinities, NaN */
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

/* --------------------------------------------- levels in one CTA (n <= 33) */
/* level l has n_l = 2^(l+1) + 1 nodes a side; SM_TOP is the level of 33 */
constexpr int SM_TOP = 4;
constexpr int SM_THREADS = 512;
constexpr int SM_TEAM = 128;   /* threads on levels of 17 nodes and fewer */
__host__ __device__ constexpr int sm_n(int l) { return (2 << l) + 1; }
__host__ __device__ constexpr int sm_below(int l) { return l == 0 ? 0 : sm_below(l - 1) + sm_n(l - 1) * sm_n(l - 1); }
/* shared image: U, F, G = h^2 F of levels 0..SM_TOP (a V-cycle's top), V,
 * R, GR = h^2 R of levels 0..SM_TOP-1 (below its top), one residual plane */
constexpr int SM_A = sm_below(SM_TOP + 1), SM_B = sm_below(SM_TOP);
constexpr int SM_WORDS = 3 * SM_A + 3 * SM_B + sm_n(SM_TOP) * sm_n(SM_TOP);

extern __shared__ __align__(16) unsigned char mg_smem[];

template <class T, int L, bool TOP>
struct Arr {
    static constexpr int n = sm_n(L), per = 1 << L;   /* nodes a side, slots a row */
    static constexpr int o = sm_below(L);
    static __device__ __forceinline__ T* u() { return reinterpret_cast<T*>(mg_smem) + (TOP ? o : 3 * SM_A + o); }
    static __device__ __forceinline__ T* f() { return reinterpret_cast<T*>(mg_smem) + (TOP ? SM_A + o : 3 * SM_A + SM_B + o); }
    static __device__ __forceinline__ T* g() { return reinterpret_cast<T*>(mg_smem) + (TOP ? 2 * SM_A + o : 3 * SM_A + 2 * SM_B + o); }
};
template <class T>
__device__ __forceinline__ T* sm_res() { return reinterpret_cast<T*>(mg_smem) + 3 * SM_A + 3 * SM_B; }

template <int L>
__device__ __forceinline__ void team_sync() {
    if (L >= SM_TOP) __syncthreads();
    else asm volatile("bar.sync 1, %0;" ::"n"(SM_TEAM) : "memory");
}
template <int L>
__device__ __forceinline__ constexpr int team_size() { return L >= SM_TOP ? SM_THREADS : SM_TEAM; }

/* one colour of a sweep (0 red, 1 black): a row has 2^L slots */
template <class T, int L, bool TOP>
__device__ __forceinline__ void sm_sweep(int color) {
    using A = Arr<T, L, TOP>;
    constexpr int n = A::n;
    T* const u = A::u();
    const T* const g = A::g();
#pragma unroll 1
    for (int t = threadIdx.x; t < (n - 2) * A::per; t += team_size<L>()) {
        const int i = (t >> L) + 1, j = 1 + ((i + 1 + color) & 1) + 2 * (t & (A::per - 1));
        if (j <= n - 2) {
            const int k = i * n + j;
            u[k] = gs_value(u[k + n], u[k - n], u[k + 1], u[k - 1], g[k]);
        }
    }
    team_sync<L>();
}

/* the points of a level below the top start at 0: red points (0 - g)/4
 * (written by whoever produced g), then the black sweep                  */
template <class T>
__device__ __forceinline__ T red_from_zero(T g) { return down_pow2<2>((T)0 - g); }

template <class T, int L, bool TOP, int START>
__device__ __forceinline__ void sm_down(T length) {
    using A = Arr<T, L, TOP>;
    using C = Arr<T, L - 1, false>;
    constexpr int n = A::n, nc = C::n, per = A::per;
    T* const u = A::u();
    const T* const f = A::f();
    const T h = length / (T)(n - 1), h2i = (T)1.0 / (h * h);
    if (START == FROM_COARSE) {
        const T* const uc = Arr<T, L - 1, true>::u();
#pragma unroll 1
        for (int t = threadIdx.x; t < (n - 2) * per; t += team_size<L>()) {
            const int i = (t >> L) + 1, j = 1 + (i & 1) + 2 * (t & (per - 1));
            if (j <= n - 2) {
                int k1, k0;
                black_pair(i, j, nc, k1, k0);
                u[i * n + j] = down_pow2<1>(uc[k1] + uc[k0]);
            }
        }
        team_sync<L>();
    }
    if (START != FROM_ZERO) sm_sweep<T, L, TOP>(0);   /* else the red points are there */
    sm_sweep<T, L, TOP>(1);
    /* residuals where the restriction reads them: all points of even rows,
     * the black points (even j) of odd rows                              */
    T* const res = sm_res<T>();
    constexpr int na = (per - 1) * 2 * per, nb = per * per;
#pragma unroll 1
    for (int t = threadIdx.x; t < na + nb; t += team_size<L>()) {
        const int s = t - na;
        const int i = s < 0 ? 2 * (t >> (L + 1)) + 2 : 2 * (s >> L) + 1;
        const int j = s < 0 ? 1 + (t & (2 * per - 1)) : 2 * (s & (per - 1)) + 2;
        if (j <= n - 2) {
            const int k = i * n + j;
            res[k] = resid_value(u[k + n], u[k - n], u[k + 1], u[k - 1], u[k], f[k], h2i);
        }
    }
    team_sync<L>();
    /* half weighting; the coarse red points get their first value here */
    const T hc = length / (T)(nc - 1), h2c = hc * hc;
    T* const rc = C::f();
    T* const gc = C::g();
    T* const vc = C::u();
#pragma unroll 1
    for (int t = threadIdx.x; t < (nc - 2) * per; t += team_size<L>()) {
        const int ic = (t >> L) + 1, jc = 1 + (t & (per - 1));
        if (jc <= nc - 2) {
            const int k = 2 * ic * n + 2 * jc, kc = ic * nc + jc;
            const T r = half_weight(res[k], res[k + n], res[k - n], res[k + 1], res[k - 1]);
            const T g = h2c * r;
            rc[kc] = r;
            gc[kc] = g;
            if (((ic + jc) & 1) == 0) vc[kc] = red_from_zero(g);
        }
    }
    team_sync<L>();
}
/* the correction of the black points, then a sweep */
template <class T, int L, bool TOP>
__device__ __forceinline__ void sm_up() {
    using A = Arr<T, L, TOP>;
    constexpr int n = A::n, per = A::per, nc = sm_n(L - 1);
    T* const u = A::u();
    const T* const vc = Arr<T, L - 1, false>::u();
#pragma unroll 1
    for (int t = threadIdx.x; t < (n - 2) * per; t += team_size<L>()) {
        const int i = (t >> L) + 1, j = 1 + (i & 1) + 2 * (t & (per - 1));
        if (j <= n - 2) {
            int k1, k0;
            black_pair(i, j, nc, k1, k0);
            u[i * n + j] = fma_t((T)0.5, vc[k1] + vc[k0], u[i * n + j]);
        }
    }
    team_sync<L>();
    sm_sweep<T, L, TOP>(0);
    sm_sweep<T, L, TOP>(1);
}
/* V-cycle with top L; entered by the team of level L */
template <class T, int L, bool TOP, int START>
struct SmV {
    static __device__ __noinline__ void run(T length) {
        sm_down<T, L, TOP, START>(length);
        if (L == SM_TOP) {
            if (threadIdx.x < SM_TEAM) SmV<T, L - 1, false, FROM_ZERO>::run(length);
            __syncthreads();
        } else {
            SmV<T, L - 1, false, FROM_ZERO>::run(length);
        }
        sm_up<T, L, TOP>();
    }
};
/* the 3x3 grid: u = -h^2 f / 4 (mglin.cpp:103-110) */
template <class T, bool TOP, int START>
struct SmV<T, 0, TOP, START> {
    static __device__ __forceinline__ void run(T length) {
        if (threadIdx.x == 0) {
            const T h = (T)0.5 * length;
            Arr<T, 0, TOP>::u()[4] = -h * h * Arr<T, 0, TOP>::f()[4] / (T)4.0;
        }
        team_sync<0>();
    }
};

/* all shared words to 0: the walls of every level stay 0 */
template <class T>
__device__ __forceinline__ void sm_clear() {
    T* const s = reinterpret_cast<T*>(mg_smem);
    for (int k = threadIdx.x; k < SM_WORDS; k += SM_THREADS) s[k] = (T)0;
    __syncthreads();
}

/* F of level L (and G) from a global right-hand side with the same nodes */
template <class T, int L>
__device__ __forceinline__ void sm_load_f(const T* gf, T length, bool red) {
    using A = Arr<T, L, true>;
    constexpr int n = A::n;
    const T h = length / (T)(n - 1), h2 = h * h;
    for (int k = threadIdx.x; k < n * n; k += SM_THREADS) {
        const int i = k / n, j = k - i * n;
        if (i > 0 && j > 0 && i < n - 1 && j < n - 1) {
            const T f = __ldcg(gf + k), g = h2 * f;
            A::f()[k] = f;
            A::g()[k] = g;
            if (red && ((i + j) & 1) == 0) A::u()[k] = red_from_zero(g);
        }
    }
    __syncthreads();
}
template <class T, int L>
__device__ __forceinline__ void sm_store_u(T* gu) {
    using A = Arr<T, L, true>;
    constexpr int n = A::n;
    for (int k = threadIdx.x; k < n * n; k += SM_THREADS) {
        const int i = k / n, j = k - i * n;
        if (i > 0 && j > 0 && i < n - 1 && j < n - 1) gu[k] = A::u()[k];
    }
    __syncthreads();
}
/* F of level L from F of level L+1 (interior) */
template <class T, int L>
__device__ __forceinline__ void sm_restrict_f(T length) {
    using A = Arr<T, L, true>;
    constexpr int n = A::n, nf = sm_n(L + 1);
    const T h = length / (T)(n - 1), h2 = h * h;
    const T* const ff = Arr<T, L + 1, true>::f();
    for (int k = threadIdx.x; k < n * n; k += SM_THREADS) {
        const int i = k / n, j = k - i * n;
        if (i > 0 && j > 0 && i < n - 1 && j < n - 1) {
            const int q = 2 * i * nf + 2 * j;
            const T f = half_weight(ff[q], ff[q + nf], ff[q - nf], ff[q + 1], ff[q - 1]);
            A::f()[k] = f;
            A::g()[k] = h2 * f;
        }
    }
    __syncthreads();
}
/* F of the levels below L, then the full multigrid up to level L */
template <class T, int L>
struct SmF {
    static __device__ __forceinline__ void restrict_all(T length) {
        sm_restrict_f<T, L - 1>(length);
        SmF<T, L - 1>::restrict_all(length);
    }
    static __device__ __forceinline__ void solve(T length) {
        SmF<T, L - 1>::solve(length);
        if (L >= SM_TOP) __syncthreads();
        if (L >= SM_TOP || threadIdx.x < SM_TEAM) {
            SmV<T, L, true, FROM_COARSE>::run(length);
            SmV<T, L, true, FROM_U>::run(length);
        }
    }
};
template <class T>
struct SmF<T, 0> {
    static __device__ __forceinline__ void restrict_all(T) {}
    static __device__ __forceinline__ void solve(T length) {
        if (threadIdx.x < SM_TEAM) SmV<T, 0, true, FROM_U>::run(length);
    }
};
/* full multigrid at level L, right-hand side f, into u (one CTA) */
template <class T, int L>
__device__ __forceinline__ void sm_fmg(const T* f, T* u, T length) {
    sm_clear<T>();
    sm_load_f<T, L>(f, length, false);
    SmF<T, L>::restrict_all(length);
    SmF<T, L>::solve(length);
    __syncthreads();
    sm_store_u<T, L>(u);
}
/* one V-cycle from 0 at level L, right-hand side f, into u (one CTA) */
template <class T, int L>
__device__ __forceinline__ void sm_vcycle0(const T* f, T* u, T length) {
    sm_clear<T>();
    sm_load_f<T, L>(f, length, true);
    if (L >= SM_TOP) {
        SmV<T, L, true, FROM_ZERO>::run(length);
    } else {
        if (threadIdx.x < SM_TEAM) SmV<T, L, true, FROM_ZERO>::run(length);
        __syncthreads();
    }
    sm_store_u<T, L>(u);
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
                                          T length) {
    using L = Tile<M, N>;
    T* const su = reinterpret_cast<T*>(mg_smem);
    T* const sf = su + L::UR * L::UC;
    T* const sr = sf + L::FR * L::FC;
    const int nc = n / 2 + 1;
    const T h = length / (T)(n - 1), h2 = h * h, h2i = (T)1.0 / (h * h);
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
__device__ __forceinline__ void tile_up(const T* w, const T* vc, const T* f, T* u, int n, int ic0, int jc0, T length) {
    constexpr int UR = 2 * M + 4, UC = 2 * N + 4, FR = 2 * M + 2, FC = 2 * N + 2;
    T* const su = reinterpret_cast<T*>(mg_smem);
    T* const sf = su + UR * UC;
    const int nc = n / 2 + 1;
    const T h = length / (T)(n - 1), h2 = h * h;
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

/* ------------------------------------ levels on the whole GPU (n >= 257) */
#define MG_M 8
#define MG_N 16
#define MG_THREADS 256
template <class T, int START>
__global__ void __launch_bounds__(MG_THREADS) k_mg_down(const T* u, const T* uc, const T* f, T* w, T* rc, int n, T length) {
    pgb_pdl_entry();
    tile_down<T, MG_M, MG_N, START, MG_THREADS>(u, uc, f, w, rc, n, 1 + MG_M * blockIdx.y, 1 + MG_N * blockIdx.x, length);
}
template <class T>
__global__ void __launch_bounds__(MG_THREADS) k_mg_up(const T* w, const T* vc, const T* f, T* u, int n, T length) {
    pgb_pdl_entry();
    tile_up<T, MG_M, MG_N, MG_THREADS>(w, vc, f, u, n, 1 + MG_M * blockIdx.y, 1 + MG_N * blockIdx.x, length);
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

/* ------------------------------------------- levels in one launch (n <= 129) */
constexpr int CL_CTAS = 16;
/* level arrays in global memory */
template <class T>
struct MgPtrs {
    T* u[PGB_MAX_LEVELS];
    T* f[PGB_MAX_LEVELS];
    T* v[PGB_MAX_LEVELS];
    T* r[PGB_MAX_LEVELS];
    T* w[PGB_MAX_LEVELS];
};

/* every CTA's global writes before are seen by every CTA's reads after */
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ int cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}

/* V-cycle of a cluster level L (5: 65 nodes, 6: 129): CTA c takes the
 * coarse rows from 1 + c M, M = 2^L / 16                                */
template <class T, int L, int START>
__device__ __forceinline__ void cl_vcycle(const MgPtrs<T>& p, T* u, const T* f, const T* uc, T length);
template <class T, int L>
struct ClLower {
    static __device__ __forceinline__ void run(const MgPtrs<T>& p, T length) {
        cl_vcycle<T, L, FROM_ZERO>(p, p.v[L], p.r[L], nullptr, length);
    }
};
template <class T>
struct ClLower<T, SM_TOP> {
    static __device__ __forceinline__ void run(const MgPtrs<T>& p, T length) {
        if (cluster_rank() == 0) sm_vcycle0<T, SM_TOP>(p.r[SM_TOP], p.v[SM_TOP], length);
        cluster_sync();
    }
};
template <class T, int L, int START>
__device__ __forceinline__ void cl_vcycle(const MgPtrs<T>& p, T* u, const T* f, const T* uc, T length) {
    constexpr int M = (1 << L) / CL_CTAS, N = 1 << L;
    const int ic0 = 1 + M * cluster_rank();
    tile_down<T, M, N, START, SM_THREADS>(u, uc, f, p.w[L], p.r[L - 1], sm_n(L), ic0, 1, length);
    cluster_sync();
    ClLower<T, L - 1>::run(p, length);
    tile_up<T, M, N, SM_THREADS>(p.w[L], p.v[L - 1], f, u, sm_n(L), ic0, 1, length);
    cluster_sync();
}
/* right-hand side of level L from level L+1, rows shared out */
template <class T, int L>
__device__ __forceinline__ void cl_restrict(const MgPtrs<T>& p) {
    constexpr int n = sm_n(L), nf = sm_n(L + 1);
    for (int k = threadIdx.x + SM_THREADS * cluster_rank(); k < n * n; k += SM_THREADS * CL_CTAS) {
        const int i = k / n, j = k - i * n;
        if (i > 0 && j > 0 && i < n - 1 && j < n - 1) {
            const T* const q = p.f[L + 1] + 2 * i * nf + 2 * j;
            p.f[L][k] = half_weight(__ldcg(q), __ldcg(q + nf), __ldcg(q - nf), __ldcg(q + 1), __ldcg(q - 1));
        }
    }
    cluster_sync();
}
template <class T, int L>
struct ClF {
    static __device__ __forceinline__ void run(const MgPtrs<T>& p, T length) {
        cl_restrict<T, L - 1>(p);
        ClF<T, L - 1>::run(p, length);
        cl_vcycle<T, L, FROM_COARSE>(p, p.u[L], p.f[L], p.u[L - 1], length);
        cl_vcycle<T, L, FROM_U>(p, p.u[L], p.f[L], nullptr, length);
    }
};
template <class T>
struct ClF<T, SM_TOP> {
    static __device__ __forceinline__ void run(const MgPtrs<T>& p, T length) {
        if (cluster_rank() == 0) sm_fmg<T, SM_TOP>(p.f[SM_TOP], p.u[SM_TOP], length);
        cluster_sync();
    }
};

/* FMG: full multigrid at level J from f[J] into u[J]; else one V-cycle
 * from 0 at level J on the right-hand side r[J] into v[J].  A cluster of
 * CL_CTAS CTAs for J > SM_TOP, one CTA otherwise.                        */
template <class T, int J, bool FMG>
__global__ void __launch_bounds__(SM_THREADS) k_mg_levels(MgPtrs<T> p, T length) {
    pgb_pdl_entry();
    if constexpr (J > SM_TOP) {
        if constexpr (FMG) ClF<T, J>::run(p, length);
        else ClLower<T, J>::run(p, length);
    } else {
        if constexpr (FMG) sm_fmg<T, J>(p.f[J], p.u[J], length);
        else sm_vcycle0<T, J>(p.r[J], p.v[J], length);
    }
}

/* ====================================================== host side */
constexpr int CL_TOP = 6;   /* the finest level of k_mg_levels (129 nodes) */
constexpr int mg_max(int a, int b) { return a > b ? a : b; }
template <class T, int J>
constexpr size_t levels_smem() {
    return sizeof(T) * (J <= SM_TOP ? SM_WORDS
                        : J == 5 ? mg_max(SM_WORDS, Tile<2, 32>::WORDS)
                                 : mg_max(SM_WORDS, mg_max(Tile<2, 32>::WORDS, Tile<4, 64>::WORDS)));
}
template <class T>
constexpr size_t tile_smem() { return sizeof(T) * Tile<MG_M, MG_N>::WORDS; }

template <class T>
MgPtrs<T> mg_ptrs(pgb_run* r);
template <>
MgPtrs<double> mg_ptrs<double>(pgb_run* r) {
    MgPtrs<double> p;
    for (int l = 0; l < PGB_MAX_LEVELS; ++l) {
        p.u[l] = r->mg_u[l]; p.f[l] = r->mg_f[l]; p.v[l] = r->mg_v[l]; p.r[l] = r->mg_r[l]; p.w[l] = r->mg_w[l];
    }
    return p;
}
template <>
MgPtrs<float> mg_ptrs<float>(pgb_run* r) {
    MgPtrs<float> p;
    for (int l = 0; l < PGB_MAX_LEVELS; ++l) {
        p.u[l] = r->mg32_u[l]; p.f[l] = r->mg32_f[l]; p.v[l] = r->mg32_v[l]; p.r[l] = r->mg32_r[l]; p.w[l] = r->mg32_w[l];
    }
    return p;
}

template <class T, int J, bool FMG>
cudaError_t levels_attr() {
    cudaError_t e = cudaFuncSetAttribute(k_mg_levels<T, J, FMG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)levels_smem<T, J>());
    if (e == cudaSuccess && J > SM_TOP)
        e = cudaFuncSetAttribute(k_mg_levels<T, J, FMG>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}
template <class T, int J, bool FMG>
int levels_go(pgb_run* r) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(J > SM_TOP ? CL_CTAS : 1);
    cfg.blockDim = dim3(SM_THREADS);
    cfg.dynamicSmemBytes = levels_smem<T, J>();
    cfg.stream = r->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CL_CTAS;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = J > SM_TOP ? 2 : 1;
    PGB_CK(r, cudaLaunchKernelEx(&cfg, k_mg_levels<T, J, FMG>, mg_ptrs<T>(r), (T)r->p.xlength));
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
        default: return levels_go<T, 6, FMG>(r);
    }
}
template <class T>
int mg_attrs(pgb_run* r) {
    PGB_CK(r, (levels_attr<T, 1, true>()));
    PGB_CK(r, (levels_attr<T, 2, true>()));
    PGB_CK(r, (levels_attr<T, 3, true>()));
    PGB_CK(r, (levels_attr<T, 4, true>()));
    PGB_CK(r, (levels_attr<T, 5, true>()));
    PGB_CK(r, (levels_attr<T, 6, true>()));
    PGB_CK(r, (levels_attr<T, 1, false>()));
    PGB_CK(r, (levels_attr<T, 2, false>()));
    PGB_CK(r, (levels_attr<T, 3, false>()));
    PGB_CK(r, (levels_attr<T, 4, false>()));
    PGB_CK(r, (levels_attr<T, 5, false>()));
    PGB_CK(r, (levels_attr<T, 6, false>()));
    return 0;
}
static_assert(tile_smem<double>() <= 48 * 1024, "the tile kernels use no more than the default shared memory");

/* V-cycle at level j > CL_TOP (mglin.cpp:176-196): u -> w -> u.  A level
 * has one V-cycle in flight at a time, so one spare buffer w serves.     */
template <class T, int START>
int vcycle(pgb_run* r, const MgPtrs<T>& p, int j, T* u, const T* f, const T* uc) {
    const int n = r->mg_n[j], nc = r->mg_n[j - 1];
    const dim3 grid((nc - 2 + MG_N - 1) / MG_N, (nc - 2 + MG_M - 1) / MG_M);
    const T length = (T)r->p.xlength;
    PGB_CK(r, pgb_launch_pdl(k_mg_down<T, START>, grid, dim3(MG_THREADS), tile_smem<T>(), r->stream, (const T*)u, uc, f,
                             p.w[j], p.r[j - 1], n, length));
    r->launches++;
    if (j - 1 > CL_TOP) {
        if (vcycle<T, FROM_ZERO>(r, p, j - 1, p.v[j - 1], p.r[j - 1], nullptr)) return PGB_ERR_CUDA;
    } else if (levels_launch<T, false>(r, j - 1)) {
        return PGB_ERR_CUDA;
    }
    PGB_CK(r, pgb_launch_pdl(k_mg_up<T>, grid, dim3(MG_THREADS), tile_smem<T>(), r->stream, (const T*)p.w[j],
                             (const T*)p.v[j - 1], f, u, n, length));
    r->launches++;
    return 0;
}

template <class T>
int fmg(pgb_run* r) {
    const int ng = r->ng;
    const MgPtrs<T> p = mg_ptrs<T>(r);
    for (int j = ng - 2; j >= CL_TOP; --j) {
        const int nc = r->mg_n[j], blocks = (nc * nc + 255) / 256;
        PGB_CK(r, pgb_launch_pdl(k_mg_restrict<T>, dim3(blocks), dim3(256), 0, r->stream, p.f[j], (const T*)p.f[j + 1], nc));
        r->launches++;
    }
    if (levels_launch<T, true>(r, ng - 1 < CL_TOP ? ng - 1 : CL_TOP)) return PGB_ERR_CUDA;
    for (int j = CL_TOP + 1; j < ng; ++j) {
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
    const int rc = top > CL_TOP ? vcycle<float, FROM_ZERO>(r, p, top, p.v[top], p.r[top], nullptr)
                                : levels_launch<float, false>(r, top);
    if (rc) return rc;
    PGB_CK(r, cudaGetLastError());
    return 0;
}
