/*
 * Grid kernels: charge finalisation and rho, the Poisson right-hand side,
 * the defect correction of the Poisson modes and the electric field.
 *
 * Reference path: particle::collect_charge edge doubling
 * (particle.cpp:829-845), fields::grid_rho (fields.cpp:100-143),
 * fields::grid_potential (fields.cpp:169-220), fields::grid_electric_field (fields.cpp:230-268).
 *
 * Compiled with --fmad=false: the FP64 right-hand side, field and defect
 * perform the reference's additions and multiplications one by one.  The
 * multigrid is in pgb_mg.cu, the sine-transform solver in pgb_dst.cu.
 */
#include <cuda_runtime.h>
#include <math.h>
#include "pgb_internal.h"
#include "pgb_fp64.cuh"

/* ------------------------------------------------ charge, rho, rhs */
enum { F32_NONE = 0, F32_CHARGE = 1, F32_RHS = 2 };
struct FinalizeArgs {
    unsigned long long* acc[2];
    double* q[2];
    double* rho;
    double* f;            /* Poisson right-hand side, or null */
    float* f32;           /* an FP32 right-hand side, by f32_what */
    int f32_what;         /* F32_CHARGE: -rho/EPSILON on the interior (the walls'
                             terms are in the wall solutions), F32_RHS: f   */
    int nx, ny;
    double qs[2];         /* qc/(DX*DY) per unit of the accumulators, per species */
    int mask;             /* species whose q is rebuilt from acc */
    int clear;            /* zero acc once read                  */
    double coef;          /* 1/EPSILON */
    double divdxdy;       /* 1/(DX*DY) */
    double phi0x, phi0y, phily;
    const double* phi_tab;   /* right wall: phi_tab[t - t_base] (fields.cpp:177) */
    const DevState* ds;
};

__device__ __forceinline__ double edge_factor(int i, int j, int nx, int ny) {
    bool ex = (i == 0 || i == nx - 1), ey = (j == 0 || j == ny - 1);
    /* columns doubled, rows doubled, corners doubled again (particle.cpp:830-845) */
    return (ex ? 2.0 : 1.0) * (ey ? 2.0 : 1.0) * ((ex && ey) ? 2.0 : 1.0);
}

/* RHS of fields::grid_potential (fields.cpp:184-204) for node (j, i) from
 * charge = -coef * rho                                                   */
__device__ __forceinline__ double rhs_node(double charge, int i, int j, const FinalizeArgs& a, double phirx) {
    double f = charge;
    if (i == 1) f = f - a.phi0x * a.divdxdy;
    if (i == a.nx - 2) f = f - phirx * a.divdxdy;
    if (j == 1) f = f - a.phi0y * a.divdxdy;
    if (j == a.ny - 2) f = f - a.phily * a.divdxdy;
    return f;
}
__device__ __forceinline__ void store_rhs(const FinalizeArgs& a, int k, int i, int j, double rho, double phirx) {
    const double charge = -a.coef * rho;
    const double f = rhs_node(charge, i, j, a, phirx);
    a.f[k] = f;
    if (a.f32_what == F32_RHS) a.f32[k] = f64_to_f32(f);
    if (a.f32_what == F32_CHARGE)
        a.f32[k] = (i > 0 && j > 0 && i < a.nx - 1 && j < a.ny - 1) ? f64_to_f32(charge) : 0.0f;
}

/* The sum is an integer number of 2^-19 of a unit weight and the edge
 * factor a power of two: q = sum * (qs * factor) rounds once, as
 * (sum * 2^-19 * qc/(DX*DY)) * factor does.                              */
__global__ void k_finalize(FinalizeArgs a) {
    pgb_pdl_entry();
    const int G = a.nx * a.ny;
    const double phirx = a.phi_tab[a.ds->tf - a.ds->t_base];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < G; k += gridDim.x * blockDim.x) {
        const long long v0 = a.mask & 1 ? (long long)a.acc[0][k] : 0, v1 = a.mask & 2 ? (long long)a.acc[1][k] : 0;
        const int j = k / a.nx, i = k - j * a.nx;
        double s0 = a.qs[0], s1 = a.qs[1];
        if (i == 0 || j == 0 || i == a.nx - 1 || j == a.ny - 1) {
            const double ef = edge_factor(i, j, a.nx, a.ny);
            s0 = s0 * ef;
            s1 = s1 * ef;
        }
        const double q0 = a.mask & 1 ? i64_to_f64(v0) * s0 : a.q[0][k];
        const double q1 = a.mask & 2 ? i64_to_f64(v1) * s1 : a.q[1][k];
        if (a.mask & 1) a.q[0][k] = q0;
        if (a.mask & 2) a.q[1][k] = q1;
        if (a.clear) a.acc[0][k] = a.acc[1][k] = 0ull;
        const double rho = q1 + q0;
        a.rho[k] = rho;
        if (a.f) store_rhs(a, k, i, j, rho, phirx);
    }
}

__global__ void k_rhs(FinalizeArgs a) {
    pgb_pdl_entry();
    const int G = a.nx * a.ny;
    const double phirx = a.phi_tab[a.ds->tf - a.ds->t_base];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < G; k += gridDim.x * blockDim.x) {
        int j = k / a.nx, i = k - j * a.nx;
        store_rhs(a, k, i, j, a.rho[k], phirx);
    }
}

/* ------------------------------------------------ potential and E field */
/* Where the potential of an interior node comes from. */
struct PhiSource {
    const double* u;      /* FP64 part, or null */
    const float* e;       /* FP32 part to add, or null */
    const double* phi;    /* or the potential itself, walls included */
};
struct FieldArgs {
    PhiSource src;
    double* phi;          /* written where src.phi is null */
    double *Ex, *Ey;      /* null: the potential only */
    float2* exy;
    int nx, ny;
    DivBy two_dx;
    double phi0x, phi0y, phily;
    const double* phi_tab;
    DevState* ds;
    int advance;          /* move the field step counter on */
};
/* the potential at node (j, i): fields.cpp:209-219 sets columns first, then
 * rows overwrite the corners                                             */
__device__ __forceinline__ double phi_at(const FieldArgs& a, double phirx, int j, int i) {
    const int k = j * a.nx + i;
    if (a.src.phi) return a.src.phi[k];
    if (j == 0) return a.phi0y;
    if (j == a.ny - 1) return a.phily;
    if (i == 0) return a.phi0x;
    if (i == a.nx - 1) return phirx;
    if (!a.src.e) return a.src.u[k];
    const double e = f32_to_f64(a.src.e[k]);
    return a.src.u ? a.src.u[k] + e : e;
}
/* fields::grid_electric_field (fields.cpp:230-268) at interior nodes, 0 on
 * the walls                                                              */
__device__ __forceinline__ double ex_interior(const FieldArgs& a, double phirx, int j, int i) {
    if (j < 1 || j > a.ny - 2 || i < 1 || i > a.nx - 2) return 0.0;
    return div_const(phi_at(a, phirx, j, i - 1) - phi_at(a, phirx, j, i + 1), a.two_dx);
}
__device__ __forceinline__ double ey_interior(const FieldArgs& a, double phirx, int j, int i) {
    if (j < 1 || j > a.ny - 2 || i < 1 || i > a.nx - 2) return 0.0;
    return div_const(phi_at(a, phirx, j - 1, i) - phi_at(a, phirx, j + 1, i), a.two_dx);
}
/* The end of a field solve in one launch: the last correction's addition,
 * the walls, E in the stride-nx layout of an (nx+1)*(ny+1) buffer (its
 * entries past nx*ny stay 0 from the allocation) and the FP32 {Ex,Ey} copy
 * read by the gather.  A block takes a 32 x 8 tile of nodes and forms each
 * potential once, in shared memory with a ring around the tile.  At 513^2 the
 * three kernels that did this took 4.0 + 3.7 + 16.5 us, most of it two FP64
 * divisions a node.                                                      */
#define FT_X 32
#define FT_Y 8
__global__ void __launch_bounds__(FT_X * FT_Y) k_field(FieldArgs a) {
    pgb_pdl_entry();
    __shared__ double s[FT_Y + 2][FT_X + 2];
    const int nx = a.nx, ny = a.ny;
    const double phirx = a.phi_tab[a.ds->tf - a.ds->t_base];
    const int i0 = blockIdx.x * FT_X - 1, j0 = blockIdx.y * FT_Y - 1;
    for (int t = threadIdx.x; t < (FT_Y + 2) * (FT_X + 2); t += FT_X * FT_Y) {
        const int r = t / (FT_X + 2), c = t - r * (FT_X + 2), j = j0 + r, i = i0 + c;
        if (j >= 0 && i >= 0 && j < ny && i < nx) s[r][c] = phi_at(a, phirx, j, i);
    }
    __syncthreads();
    const int c = threadIdx.x % FT_X + 1, r = threadIdx.x / FT_X + 1, i = i0 + c, j = j0 + r;
    if (i < nx && j < ny) {
        const int k = j * nx + i;
        if (!a.src.phi) a.phi[k] = s[r][c];
        if (a.Ex) {
            double ex, ey;
            if (i > 0 && j > 0 && i < nx - 1 && j < ny - 1) {
                ex = div_const(s[r][c - 1] - s[r][c + 1], a.two_dx);
                ey = div_const(s[r - 1][c] - s[r + 1][c], a.two_dx);
            } else {
                if (i == 0) ex = 2.0 * ex_interior(a, phirx, j, 1) - ex_interior(a, phirx, j, 2);
                else if (i == nx - 1) ex = 2.0 * ex_interior(a, phirx, j, nx - 2) - ex_interior(a, phirx, j, nx - 3);
                else ex = ex_interior(a, phirx, j, i);
                if (j == 0) ey = 2.0 * ey_interior(a, phirx, 1, i) - ey_interior(a, phirx, 2, i);
                else if (j == ny - 1) ey = 2.0 * ey_interior(a, phirx, ny - 2, i) - ey_interior(a, phirx, ny - 3, i);
                else ey = ey_interior(a, phirx, j, i);
            }
            a.Ex[k] = ex;
            a.Ey[k] = ey;
            a.exy[k] = make_float2(f64_to_f32(ex), f64_to_f32(ey));
        }
    }
    /* the last block to get here moves the field step counter on: every
     * block has read it by then                                          */
    if (a.advance) {
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&a.ds->ticket_f, 1u) == gridDim.x * gridDim.y - 1) {
                a.ds->ticket_f = 0u;
                a.ds->tf += 1;
            }
        }
    }
}

/* ---------------------------------------------- FP64 defect correction */
/* One update of the FP64 solution, u' = u + e (u' = e where u is null;
 * FIRST: u' = wc + phi_right(t) wr + e, the walls' solutions and the FP32
 * solve of the charge term), written to a second buffer so that neighbours
 * read the old values, and the FP64 defect d = f - L u' of the interior
 * (zero on the walls) stored as FP32 for the next FP32 correction.  The
 * walls of u, e and so u' are 0.  A block forms each u' of its 32 x 8 tile
 * and the ring around it once, in shared memory.  4 u' is exact, so one
 * fused operation subtracts it from the neighbours' sum as the two separate
 * ones do.  At 513^2: 17.8 (FIRST) and 12.2 us before, in FP64 operations
 * of five sums per node.                                                 */
template <bool FIRST>
__global__ void __launch_bounds__(FT_X * FT_Y) k_dc_update(const double* __restrict__ u, const double* __restrict__ wc,
                                                          const double* __restrict__ wr, const double* phi_tab,
                                                          const DevState* ds, const float* __restrict__ e,
                                                          double* __restrict__ uout, const double* __restrict__ f,
                                                          float* __restrict__ d, int n, double h2i) {
    pgb_pdl_entry();
    __shared__ double s[FT_Y + 2][FT_X + 2];
    const double phirx = FIRST ? phi_tab[ds->tf - ds->t_base] : 0.0;
    const int i0 = blockIdx.y * FT_Y - 1, j0 = blockIdx.x * FT_X - 1;
    for (int t = threadIdx.x; t < (FT_Y + 2) * (FT_X + 2); t += FT_X * FT_Y) {
        const int r = t / (FT_X + 2), c = t - r * (FT_X + 2), i = i0 + r, j = j0 + c;
        if (i >= 0 && j >= 0 && i < n && j < n) {
            const int k = i * n + j;
            const double ek = f32_to_f64(e[k]);
            s[r][c] = FIRST ? (wc[k] + phirx * wr[k]) + ek : u ? u[k] + ek : ek;
        }
    }
    __syncthreads();
    const int c = threadIdx.x % FT_X + 1, r = threadIdx.x / FT_X + 1, i = i0 + r, j = j0 + c;
    if (i >= n || j >= n) return;
    const int k = i * n + j;
    const double x = s[r][c];
    float v = 0.0f;
    if (i > 0 && j > 0 && i < n - 1 && j < n - 1)
        v = f64_to_f32(f[k] - h2i * __fma_rn(-4.0, x, s[r + 1][c] + s[r - 1][c] + s[r][c + 1] + s[r][c - 1]));
    uout[k] = x;
    d[k] = v;
}
/* ====================================================== host side */
static FinalizeArgs fin_args(pgb_run* r, int mask, bool rhs) {
    FinalizeArgs a;
    a.acc[0] = r->qacc[0]; a.acc[1] = r->qacc[1];
    a.q[0] = r->q[0]; a.q[1] = r->q[1];
    a.rho = r->rho; a.f = rhs ? r->mg_f[r->ng - 1] : nullptr;
    a.nx = r->nx; a.ny = r->ny;
    for (int s = 0; s < 2; ++s) a.qs[s] = r->sp[s].qc / (r->dx * r->dy) * (1.0 / PGB_FIX_SCALE);
    /* the FP32 solvers' right-hand side comes with the FP64 one */
    a.f32 = r->mg32_f[r->ng - 1];
    a.f32_what = !rhs || r->p.poisson_mode == PGB_POISSON_FMG_REF ? F32_NONE
                 : r->p.poisson_mode == PGB_POISSON_DST_DC        ? F32_CHARGE
                                                                  : F32_RHS;
    a.mask = mask;
    a.clear = 0;
    a.coef = 1.0 / 8.854e-12;
    a.divdxdy = 1.0 / (r->dx * r->dy);
    a.phi0x = r->p.phi_left; a.phi0y = r->p.phi_bottom; a.phily = r->p.phi_top;
    a.phi_tab = r->phi_tab; a.ds = r->ds;
    return a;
}

int pgb_launch_finalize(pgb_run* r, int mask, bool make_rhs, bool clear) {
    FinalizeArgs a = fin_args(r, mask, make_rhs);
    a.clear = clear;
    int G = r->nx * r->ny;
    PGB_CK(r, pgb_launch_pdl(k_finalize, dim3((G + 255) / 256), dim3(256), 0, r->stream, a));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_rhs(pgb_run* r) {
    FinalizeArgs a = fin_args(r, 0, true);
    int G = r->nx * r->ny;
    PGB_CK(r, pgb_launch_pdl(k_rhs, dim3((G + 255) / 256), dim3(256), 0, r->stream, a));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

static int blocks_for(long long work) {
    long long b = (work + 255) / 256;
    if (b < 1) b = 1;
    if (b > 65535) b = 65535;
    return (int)b;
}

/* the walls' terms of the right-hand side alone (rhs_node at rho = 0) */
__global__ void k_wall_rhs(FinalizeArgs a, double phirx) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.nx * a.ny; k += gridDim.x * blockDim.x) {
        int j = k / a.nx, i = k - j * a.nx;
        a.f[k] = rhs_node(-0.0, i, j, a, phirx);
    }
}
__global__ void k_to32(float* d, const double* s, int count) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) d[k] = (float)s[k];
}
/* u + e in FP64 */
__global__ void k_dc_sum(double* __restrict__ out, const double* __restrict__ u, const float* __restrict__ e, int count) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) out[k] = u[k] + (double)e[k];
}

static dim3 field_grid(int nx, int ny) { return dim3((nx + FT_X - 1) / FT_X, (ny + FT_Y - 1) / FT_Y); }

/* FP64 defect correction around an FP32 solve of L u = f64 (zero walls),
 * `passes` solves in all.  *out: the parts whose sum is the solution.
 * The FP32 solve goes from f32 to e32.                                   */
template <class Solve>
static int defect_correction(pgb_run* r, const double* f64, float* f32, const float* e32, int passes, Solve solve,
                             PhiSource* out) {
    const int n = r->nx;
    const double h = r->p.xlength / (n - 1), h2i = 1.0 / (h * h);
    double* ua = const_cast<double*>(out->u);   /* FP64 solution so far (null: 0) */
    for (int it = 1; it < passes; ++it) {
        double* const ub = ua == r->dc_u ? r->dc_u2 : r->dc_u;
        PGB_CK(r, pgb_launch_pdl(k_dc_update<false>, field_grid(n, n), dim3(FT_X * FT_Y), 0, r->stream, (const double*)ua,
                                 (const double*)nullptr, (const double*)nullptr, (const double*)nullptr,
                                 (const DevState*)nullptr, out->e, ub, f64, f32, n, h2i));
        r->launches++;
        ua = ub;
        if (solve()) return PGB_ERR_CUDA;
        *out = PhiSource{ua, e32, nullptr};
    }
    return 0;
}

/* DST_DC.  The FP32 right-hand side is in mg32_f[top].
 * lift: the first approximation is the walls' solution wc + phi_right(t) wr
 * plus the FP32 solve of the charge term alone, which keeps the walls'
 * terms (-phi/(DX DY) next to a wall, a thousand times the charge term at
 * 1 V) out of the FP32 transform, whose rounding they would otherwise
 * spread over every mode; each pass then divides the error by about 1e6
 * instead of about 300.  Otherwise the first solve is of f64 itself.  */
static int dst_dc(pgb_run* r, const double* f64, int passes, bool lift, PhiSource* out) {
    const int top = r->ng - 1, n = r->nx;
    float* const f32 = r->mg32_f[top];   /* right-hand side, then each defect */
    float* const e32 = r->mg32_u[top];   /* each FP32 solve                   */
    auto solve = [&] { return pgb_dst_solve(r, f32, e32); };
    if (solve()) return PGB_ERR_CUDA;
    *out = PhiSource{nullptr, e32, nullptr};
    if (lift) {
        const double h = r->p.xlength / (n - 1), h2i = 1.0 / (h * h);
        PGB_CK(r, pgb_launch_pdl(k_dc_update<true>, field_grid(n, n), dim3(FT_X * FT_Y), 0, r->stream, (const double*)nullptr,
                                 (const double*)r->dst_wc, (const double*)r->dst_wr, (const double*)r->phi_tab,
                                 (const DevState*)r->ds, (const float*)e32, r->dc_u, f64, f32, n, h2i));
        r->launches++;
        *out = PhiSource{r->dc_u, nullptr, nullptr};
        if (passes <= 1) return 0;
        if (solve()) return PGB_ERR_CUDA;
        out->e = e32;
        passes--;
    }
    return defect_correction(r, f64, f32, e32, passes, solve, out);
}

/* DST_DC's wall solutions: L u = (the walls' right-hand side terms), the
 * left, bottom and top walls at their potentials, then the right wall at
 * 1 V, each to FP64 rounding (eight passes; about 300x each without lift) */
static int dst_wall_solutions(pgb_run* r) {
    const size_t G = (size_t)r->nx * r->ny;
    PGB_CK(r, cudaMalloc(&r->dst_wc, G * sizeof(double)));
    PGB_CK(r, cudaMalloc(&r->dst_wr, G * sizeof(double)));
    PGB_CK(r, cudaDeviceSynchronize());   /* the setup's memsets ran on the legacy stream */
    double* const f64 = r->mg_w[r->ng - 1];   /* FP64 scratch of the top level */
    const dim3 gb(blocks_for((long long)G)), tb(256);
    for (int w = 0; w < 2; ++w) {
        FinalizeArgs a = fin_args(r, 0, true);
        a.f = f64;
        if (w == 1) a.phi0x = a.phi0y = a.phily = 0.0;
        PGB_CK(r, pgb_launch_pdl(k_wall_rhs, gb, tb, 0, r->stream, a, w == 1 ? 1.0 : 0.0));
        PGB_CK(r, pgb_launch_pdl(k_to32, gb, tb, 0, r->stream, r->mg32_f[r->ng - 1], (const double*)f64, (int)G));
        PhiSource src;
        if (dst_dc(r, f64, 8, false, &src)) return PGB_ERR_CUDA;
        PGB_CK(r, pgb_launch_pdl(k_dc_sum, gb, tb, 0, r->stream, w == 0 ? r->dst_wc : r->dst_wr, src.u, src.e, (int)G));
    }
    PGB_CK(r, cudaMemsetAsync(f64, 0, G * sizeof(double), r->stream));   /* the level's walls stay 0 */
    PGB_CK(r, cudaStreamSynchronize(r->stream));
    return 0;
}

int pgb_mg_setup(pgb_run* r) {
    for (int l = 0; l < r->ng; ++l) {
        size_t n2 = (size_t)r->mg_n[l] * r->mg_n[l];
        PGB_CK(r, cudaMalloc(&r->mg32_u[l], n2 * sizeof(float)));
        PGB_CK(r, cudaMalloc(&r->mg32_f[l], n2 * sizeof(float)));
        PGB_CK(r, cudaMalloc(&r->mg32_v[l], n2 * sizeof(float)));
        PGB_CK(r, cudaMalloc(&r->mg32_r[l], n2 * sizeof(float)));
        PGB_CK(r, cudaMalloc(&r->mg_w[l], n2 * sizeof(double)));
        PGB_CK(r, cudaMalloc(&r->mg32_w[l], n2 * sizeof(float)));
    }
    for (int l = 0; l < r->ng; ++l) {
        size_t n2 = (size_t)r->mg_n[l] * r->mg_n[l];
        PGB_CK(r, cudaMemset(r->mg_u[l], 0, n2 * sizeof(double)));
        PGB_CK(r, cudaMemset(r->mg_v[l], 0, n2 * sizeof(double)));
        PGB_CK(r, cudaMemset(r->mg32_u[l], 0, n2 * sizeof(float)));
        PGB_CK(r, cudaMemset(r->mg32_v[l], 0, n2 * sizeof(float)));
        PGB_CK(r, cudaMemset(r->mg_w[l], 0, n2 * sizeof(double)));   /* walls stay 0 */
        PGB_CK(r, cudaMemset(r->mg32_w[l], 0, n2 * sizeof(float)));
    }
    size_t G = (size_t)r->nx * r->ny;
    PGB_CK(r, cudaMalloc(&r->dc_u, G * sizeof(double)));
    PGB_CK(r, cudaMalloc(&r->dc_u2, G * sizeof(double)));
    if (pgb_mg_attributes(r)) return PGB_ERR_CUDA;
    if (r->p.poisson_mode == PGB_POISSON_DST_DC) {
        if (pgb_dst_setup(r)) return PGB_ERR_CUDA;
        if (pgb_dst_ok(r) && dst_wall_solutions(r)) return PGB_ERR_CUDA;
    }
    return 0;
}

void pgb_mg_free(pgb_run* r) {
    for (int l = 0; l < r->ng; ++l) {
        cudaFree(r->mg32_u[l]); cudaFree(r->mg32_f[l]); cudaFree(r->mg32_v[l]); cudaFree(r->mg32_r[l]);
        cudaFree(r->mg_w[l]); cudaFree(r->mg32_w[l]);
    }
    cudaFree(r->dc_u);
    cudaFree(r->dc_u2);
    cudaFree(r->dst_wc);
    cudaFree(r->dst_wr);
    pgb_dst_free(r);
}

/* fields::grid_potential after the right-hand side is in mg_f[ng-1]:
 *   FMG_REF  FP64 full multigrid with the reference's schedule (bitwise)
 *   FMG32    the same schedule in FP32
 *   FP32_DC  FP64 defect correction around FP32 multigrid: the FMG32 pass
 *            on the right-hand side, then dc_max_iters - 1 passes of
 *            (FP64 defect of the FP64 solution, one FP32 V-cycle on it
 *            from zero, FP64 addition of that correction).  The FP32 pass
 *            leaves an error of a few 1e-5 of phi; each V-cycle divides it
 *            by about ten, down to the FP64 discrete solution.
 *   DST_DC   the same FP64 defect correction around the FP32 sine-transform
 *            solve (pgb_dst.cu), which solves the discrete system exactly
 *            up to FP32 rounding (about 1e-6 of phi): a first solve, then
 *            dc_max_iters - 1 corrections, each dividing the error by
 *            about 1e6.                                                  */
static int launch_field(pgb_run* r, const PhiSource& src, bool field, bool advance) {
    FieldArgs a;
    a.src = src;
    a.phi = r->phi;
    a.Ex = field ? r->ex : nullptr;
    a.Ey = r->ey;
    a.exy = r->exy;
    a.nx = r->nx; a.ny = r->ny;
    a.two_dx = div_by(2.0 * r->dx);
    a.phi0x = r->p.phi_left; a.phi0y = r->p.phi_bottom; a.phily = r->p.phi_top;
    a.phi_tab = r->phi_tab; a.ds = r->ds;
    a.advance = advance;
    PGB_CK(r, pgb_launch_pdl(k_field, field_grid(r->nx, r->ny), dim3(FT_X * FT_Y), 0, r->stream, a));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_poisson_solve(pgb_run* r, bool field, bool advance) {
    const int top = r->ng - 1;
    PhiSource src{nullptr, nullptr, nullptr};
    if (r->p.poisson_mode == PGB_POISSON_FMG_REF) {
        if (pgb_mg_fmg64(r)) return PGB_ERR_CUDA;
        src.u = r->mg_u[top];
    } else if (r->p.poisson_mode == PGB_POISSON_DST_DC) {
        if (!pgb_dst_ok(r)) return PGB_ERR_CUDA;
        if (dst_dc(r, r->mg_f[top], r->p.dc_max_iters > 1 ? r->p.dc_max_iters : 1, true, &src)) return PGB_ERR_CUDA;
    } else {
        if (pgb_mg_fmg32(r)) return PGB_ERR_CUDA;
        src.e = r->mg32_u[top];   /* the FMG pass's result */
        const int passes = r->p.poisson_mode == PGB_POISSON_FP32_DC && r->p.dc_max_iters > 1 ? r->p.dc_max_iters : 1;
        /* each defect goes to the level's residual array, its V-cycle from 0
         * to the level's correction array                                */
        if (defect_correction(r, r->mg_f[top], r->mg32_r[top], r->mg32_v[top], passes, [&] { return pgb_mg_vcycle32(r); },
                              &src))
            return PGB_ERR_CUDA;
    }
    return launch_field(r, src, field, advance);
}

/* E of the potential in r->phi (the step's field comes with its potential) */
int pgb_launch_efield(pgb_run* r) { return launch_field(r, PhiSource{nullptr, nullptr, r->phi}, true, false); }
