/*
 * FP32 Poisson solve by discrete sine transforms (the DST_DC mode's inner
 * solver).
 *
 * fields::grid_potential solves the 5-point discrete Poisson equation
 *   (u[i+1][j] + u[i-1][j] + u[i][j+1] + u[i][j-1] - 4 u[i][j]) / h^2 = f[i][j]
 * on the interior of an n x n grid with u = 0 on the walls (mglin.cpp:
 * 116-127 relaxes exactly this system; the walls' potentials are applied
 * afterwards).  With n = N + 1 nodes and N a power of two, the sine modes
 * sin(pi j k / N) sin(pi i l / N), 1 <= k, l <= N-1, are its eigenvectors,
 * with eigenvalues -(s_k + s_l) / h^2, s_k = 4 sin^2(pi k / 2N).  So
 *   u = (2/N)^2 DST( DST(f) * (-h^2) / (s_k + s_l) )
 * with DST the type-I sine transform along each axis,
 *   S_k = sum_{j=1}^{N-1} x_j sin(pi j k / N),
 * which is its own inverse up to the factor 2/N.  This is the exact
 * discrete solution that the multigrid approaches, up to FP32 rounding
 * (about 1e-6 of phi); an FP64 defect correction around it
 * (pgb_poisson_solve) removes that.
 *
 * A type-I sine transform of length N-1 is read off a complex FFT of
 * length M = 2N of the odd extension y = (0, x_1..x_{N-1}, 0, -x_{N-1}..
 * -x_1): Y_k = -2i S_k.  Two real sequences a, b share one FFT as
 * z = y_a + i y_b: Re Z_k = 2 S_b,k and Im Z_k = -2 S_a,k.  Three launches:
 *   k_dst_rows     row pairs (i, i+1): transform over j, stored transposed
 *                  t[k-1][i-1] (rows of N floats) for the next pass
 *   k_dst_columns  pairs of k: transform over i, division by the
 *                  eigenvalue, inverse transform over l
 *   k_dst_back     row pairs: inverse transform over k, written to u
 * Each CTA runs FFTs of length M in shared memory: radix-2 butterflies,
 * decimation in time, one or two stages at a time in registers, twiddles
 * from a table made in FP64 on the host.  How many stages a pass takes does
 * not change a value.
 */
#include <cuda_runtime.h>
#include <math.h>
#include <vector>
#include "pgb_internal.h"

struct DstArgs {
    const float* f;      /* n x n right-hand side (walls not read)       */
    float* u;            /* n x n solution (walls written 0)             */
    float* t;            /* (N-1) rows of N floats                       */
    const float2* tw;    /* M/2 twiddles exp(-2 pi i q / M)              */
    const float* s;      /* N values s_k = 4 sin^2(pi k / 2N)            */
    int n, N, logM;
    float scale;         /* -(2/N)^2 h^2                                 */
};

/* Where element i of an FFT buffer, or of the twiddles, lies: bits 0-3 (a
 * bank of 8 bytes) exclusive-or bits 4 and up, folded so that the strided
 * accesses of the passes (elements M/16, 16 or 4 apart, twiddles a power of
 * two apart) spread over the banks.  Linear over GF(2): for i and
 * j without a common bit, slot(i + j) = slot(i) ^ slot(j).               */
__device__ __forceinline__ int slot(int i) {
    const int s = i >> 4;
    return i ^ ((((s & 3) << 2) ^ (s >> 2) ^ (s >> 6)) & 15);
}

/* stages s .. s + R - 1 on the 2^R elements pos + j 2^s of one thread */
template <int R>
__device__ __forceinline__ void fft_stages(float2 (&v)[1 << R], const float2* stw, int pos, int s, int logM) {
#pragma unroll
    for (int q = 0; q < R; ++q) {
#pragma unroll
        for (int m = 0; m < (1 << q); ++m) {
            const float2 w = stw[slot((pos + (m << s)) << (logM - 1 - s - q))];
#pragma unroll
            for (int p = m; p < (1 << R); p += 2 << q) {
                const float2 a = v[p], c = v[p + (1 << q)];
                const float2 tt = make_float2(w.x * c.x - w.y * c.y, w.x * c.y + w.y * c.x);
                v[p] = make_float2(a.x + tt.x, a.y + tt.y);
                v[p + (1 << q)] = make_float2(a.x - tt.x, a.y - tt.y);
            }
        }
    }
}
/* one pass of R stages over z; the last one hands Z_k, k < M/2, to put */
template <int R, class P>
__device__ __forceinline__ void fft_pass(float2* z, const float2* stw, int s, int logM, P put) {
    const bool last = s + R == logM;
    for (int t = threadIdx.x; t < 1 << (logM - R); t += blockDim.x) {
        const int pos = t & ((1 << s) - 1), base = ((t >> s) << (s + R)) + pos, b = slot(base);
        float2 v[1 << R];
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) v[j] = z[b ^ slot(j << s)];
        fft_stages<R>(v, stw, pos, s, logM);
        if (last) {
#pragma unroll
            for (int j = 0; j < (1 << R) / 2; ++j) put(base + (j << s), v[j]);
        } else {
#pragma unroll
            for (int j = 0; j < (1 << R); ++j) z[b ^ slot(j << s)] = v[j];
        }
    }
    __syncthreads();
}
/* FFT of length M = 2^logM of the odd extension of the pair (a_q, b_q) =
 * get(q), q = 1..N-1: radix-2 butterflies, decimation in time, R stages at
 * a time in registers; put(k, Z_k) for k < N.  The first pass takes its
 * elements (t, t + M/2^R, ... in order, as the bit reversal wants them)
 * straight from get.                                                     */
template <int R, class G, class P>
__device__ __forceinline__ void fft_odd(float2* z, const float2* stw, int N, int logM, G get, P put) {
    const int M = 2 * N;
    for (int t = threadIdx.x; t < M >> R; t += blockDim.x) {
        float2 v[1 << R];
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) {
            const int q = t + (int)(__brev((unsigned)j) >> (32 - R)) * (M >> R);
            v[j] = make_float2(0.0f, 0.0f);
            if (q > 0 && q < N) v[j] = get(q);
            else if (q > N) {
                const float2 x = get(M - q);
                v[j] = make_float2(-x.x, -x.y);
            }
        }
        fft_stages<R>(v, stw, 0, 0, logM);
        const int b = slot((int)(((unsigned long long)__brev((unsigned)t) << (logM - R)) >> 32) << R);
#pragma unroll
        for (int j = 0; j < (1 << R); ++j) z[b ^ slot(j)] = v[j];
    }
    __syncthreads();
    int s = R;
    for (; s + R < logM; s += R) fft_pass<R>(z, stw, s, logM, put);
    if (logM - s == R) fft_pass<R>(z, stw, s, logM, put);
    else fft_pass<1>(z, stw, s, logM, put);
}

__device__ __forceinline__ float2* dst_smem(float2*& stw, int M) {
    extern __shared__ __align__(16) float2 smem[];
    stw = smem;              /* M/2 twiddles */
    return smem + M / 2;     /* then the FFT buffer, M, and N coefficients */
}

__device__ __forceinline__ void stage_twiddles(float2* stw, const float2* tw, int M) {
    for (int q = threadIdx.x; q < M / 2; q += blockDim.x) stw[slot(q)] = tw[q];
}

/* row pair p: rows i0 = 2p+1 and i0+1 (the wall row n-1 reads as 0) */
template <int R>
__global__ void k_dst_rows(DstArgs a) {
    const int N = a.N, M = 2 * N, n = a.n;
    float2* stw;
    float2* z = dst_smem(stw, M);
    stage_twiddles(stw, a.tw, M);   /* the run's own table: no kernel before writes it */
    pgb_pdl_entry();
    __syncthreads();
    const int i0 = 2 * blockIdx.x + 1, i1 = i0 + 1;
    const float* ra = a.f + (size_t)i0 * n;
    const float* rb = i1 <= n - 2 ? a.f + (size_t)i1 * n : nullptr;
    /* S_a,k = -Im Z_k / 2 (row i0), S_b,k = Re Z_k / 2 (row i1); for the
     * wall row an exact 0, not the rounding of row i0 that Re Z_k holds  */
    fft_odd<R>(z, stw, N, a.logM, [&](int j) { return make_float2(ra[j], rb ? rb[j] : 0.0f); },
               [&](int k, float2 Z) {
                   if (k > 0)
                       *reinterpret_cast<float2*>(a.t + (size_t)(k - 1) * N + (i0 - 1)) =
                           make_float2(-0.5f * Z.y, rb ? 0.5f * Z.x : 0.0f);
               });
}

/* pair q of frequencies k0 = 2q+1, k1 = k0+1 (k1 = N reads as 0, not written) */
template <int R>
__global__ void k_dst_columns(DstArgs a) {
    const int N = a.N, M = 2 * N;
    float2* stw;
    float2* z = dst_smem(stw, M);
    float2* const coef = z + M;
    stage_twiddles(stw, a.tw, M);
    pgb_pdl_entry();
    __syncthreads();
    const int k0 = 2 * blockIdx.x + 1, k1 = k0 + 1;
    float* const ta = a.t + (size_t)(k0 - 1) * N;
    float* const tb = k1 <= N - 1 ? a.t + (size_t)(k1 - 1) * N : nullptr;
    const float sa = a.s[k0], sb = a.s[k1 < N ? k1 : 1];
    /* the solution's coefficients, then the transform of those over l */
    fft_odd<R>(z, stw, N, a.logM, [&](int i) { return make_float2(ta[i - 1], tb ? tb[i - 1] : 0.0f); },
               [&](int l, float2 Z) {
                   if (l == 0) return;
                   const float sl = a.s[l];
                   coef[l] = make_float2((-0.5f * Z.y) * a.scale / (sa + sl), tb ? (0.5f * Z.x) * a.scale / (sb + sl) : 0.0f);
               });
    fft_odd<R>(z, stw, N, a.logM, [&](int l) { return coef[l]; },
               [&](int i, float2 Z) {
                   if (i == 0) return;
                   ta[i - 1] = -0.5f * Z.y;
                   if (tb) tb[i - 1] = 0.5f * Z.x;
               });
}

/* row pair p: u rows i0 = 2p+1 and i0+1 from t's columns i0-1 and i0 */
template <int R>
__global__ void k_dst_back(DstArgs a) {
    const int N = a.N, M = 2 * N, n = a.n;
    float2* stw;
    float2* z = dst_smem(stw, M);
    stage_twiddles(stw, a.tw, M);
    pgb_pdl_entry();
    __syncthreads();
    const int i0 = 2 * blockIdx.x + 1, i1 = i0 + 1;
    /* the wall row's slot (column N-1 of t) is never written by the column
     * pass: read it as 0, or its values would leak into row i0 through the
     * rounding of the shared transform                                    */
    const bool wall = i1 > n - 2;
    float* const ua = a.u + (size_t)i0 * n;
    float* const ub = a.u + (size_t)i1 * n;   /* i1 <= n-1: the top wall row is written 0 */
    fft_odd<R>(z, stw, N, a.logM,
               [&](int k) {
                   const float2 v = *reinterpret_cast<const float2*>(a.t + (size_t)(k - 1) * N + (i0 - 1));
                   return make_float2(v.x, wall ? 0.0f : v.y);
               },
               [&](int j, float2 Z) {
                   ua[j] = j > 0 ? -0.5f * Z.y : 0.0f;
                   ub[j] = j > 0 && !wall ? 0.5f * Z.x : 0.0f;
                   if (blockIdx.x == 0) a.u[j] = 0.0f;   /* the bottom wall row */
                   if (j == 0) {                         /* the right walls */
                       ua[N] = ub[N] = 0.0f;
                       if (blockIdx.x == 0) a.u[N] = 0.0f;
                   }
               });
}

static int dst_threads(int per) { return per < 32 ? 32 : (per > 512 ? 512 : per); }

template <int R>
static int dst_attributes(pgb_run* r, int smem) {
    PGB_CK(r, cudaFuncSetAttribute(k_dst_rows<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    PGB_CK(r, cudaFuncSetAttribute(k_dst_columns<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    PGB_CK(r, cudaFuncSetAttribute(k_dst_back<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    return 0;
}
template <int R>
static int dst_launch(pgb_run* r, const DstArgs& a) {
    const int M = 2 * a.N;
    const dim3 th(dst_threads(M >> R)), blocks(a.N / 2);
    const size_t sm1 = sizeof(float2) * (M / 2 + M), sm2 = sm1 + sizeof(float2) * a.N;
    PGB_CK(r, pgb_launch_pdl(k_dst_rows<R>, blocks, th, sm1, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_dst_columns<R>, blocks, th, sm2, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_dst_back<R>, blocks, th, sm1, r->stream, a));
    r->launches += 3;
    PGB_CK(r, cudaGetLastError());
    return 0;
}
/* Stages per pass: one point pair a thread is the shorter chain where the
 * kernels are launch and latency, two stages in registers halve the traffic
 * with shared memory and the barriers where they are not.  A pass of the
 * solver (three kernels and the FP64 update), R = 1 / 2 / 3, and before
 * (radix-2 in place from a bit-reversed store, up to 16-way bank conflicts
 * on it and on the twiddles): 65 nodes 10.2 / 11.9 / 14.4 (10.9) us,
 * 129 12.1 / 13.3 / 18.1 (12.8), 257 14.6 / 14.9 / 19.7 (16.1),
 * 513 28.7 / 23.3 / 25.6 (34.5).  At 257 other kernels run beside it, so
 * there the one with fewer instructions.                                 */
static bool dst_two_stages(int M) { return M >= 512; }

int pgb_dst_setup(pgb_run* r) {
    const int n = r->nx, N = n - 1;
    if (n != r->ny || N < 4 || (N & (N - 1))) return 0;   /* not a (2^k+1)^2 grid: the mode is refused at solve time */
    const int M = 2 * N;
    std::vector<float2> tw(M / 2);
    for (int q = 0; q < M / 2; ++q) {
        const double ang = -2.0 * M_PI * (double)q / (double)M;
        tw[q] = make_float2((float)cos(ang), (float)sin(ang));
    }
    std::vector<float> s(N);
    for (int k = 0; k < N; ++k) {
        const double v = sin(M_PI * (double)k / (2.0 * N));
        s[k] = (float)(4.0 * v * v);
    }
    PGB_CK(r, cudaMalloc(&r->dst_tw, sizeof(float2) * tw.size()));
    PGB_CK(r, cudaMalloc(&r->dst_s, sizeof(float) * s.size()));
    PGB_CK(r, cudaMalloc(&r->dst_t, sizeof(float) * (size_t)(N - 1) * N));
    PGB_CK(r, cudaMemcpy(r->dst_tw, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice));
    PGB_CK(r, cudaMemcpy(r->dst_s, s.data(), sizeof(float) * s.size(), cudaMemcpyHostToDevice));
    const int smem = (int)(sizeof(float2) * (M / 2 + 2 * M));
    if (smem > 48 * 1024 && dst_attributes<2>(r, smem)) return PGB_ERR_CUDA;
    return 0;
}

void pgb_dst_free(pgb_run* r) {
    cudaFree(r->dst_tw);
    cudaFree(r->dst_s);
    cudaFree(r->dst_t);
    r->dst_tw = nullptr;
    r->dst_s = nullptr;
    r->dst_t = nullptr;
}

bool pgb_dst_ok(const pgb_run* r) { return r->dst_t != nullptr; }

/* u = the FP32 solution of L u = f with zero walls (f's walls not read) */
int pgb_dst_solve(pgb_run* r, const float* f, float* u) {
    if (!r->dst_t) return PGB_ERR_CUDA;
    DstArgs a;
    a.f = f; a.u = u; a.t = r->dst_t; a.tw = r->dst_tw; a.s = r->dst_s;
    a.n = r->nx; a.N = r->nx - 1;
    const int M = 2 * a.N;
    a.logM = 0;
    while ((1 << a.logM) < M) a.logM++;
    const double h = r->p.xlength / (double)a.N;
    a.scale = (float)(-(2.0 / a.N) * (2.0 / a.N) * h * h);
    return dst_two_stages(M) ? dst_launch<2>(r, a) : dst_launch<1>(r, a);
}
