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

/* ------------------------------------------------ charge, rho, rhs */
struct FinalizeArgs {
    unsigned long long* acc[2];
    double* q[2];
    double* rho;
    double* f;            /* Poisson right-hand side, or null */
    int nx, ny;
    double qcdxdy[2];     /* qc/(DX*DY) per species */
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

/* RHS of fields::grid_potential (fields.cpp:184-204) for node (j, i) */
__device__ __forceinline__ double rhs_node(double rho, int i, int j, const FinalizeArgs& a, double phirx) {
    double f = -a.coef * rho;
    if (i == 1) f = f - a.phi0x * a.divdxdy;
    if (i == a.nx - 2) f = f - phirx * a.divdxdy;
    if (j == 1) f = f - a.phi0y * a.divdxdy;
    if (j == a.ny - 2) f = f - a.phily * a.divdxdy;
    return f;
}

__global__ void k_finalize(FinalizeArgs a) {
    pgb_pdl_entry();
    const int G = a.nx * a.ny;
    const double phirx = a.phi_tab[a.ds->tf - a.ds->t_base];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < G; k += gridDim.x * blockDim.x) {
        int j = k / a.nx, i = k - j * a.nx;
        double ef = edge_factor(i, j, a.nx, a.ny);
        for (int s = 0; s < 2; ++s)
            if (a.mask & (1 << s)) {
                double v = (double)(long long)a.acc[s][k] * (1.0 / PGB_FIX_SCALE);
                if (a.clear) a.acc[s][k] = 0ull;
                a.q[s][k] = (v * a.qcdxdy[s]) * ef;
            }
        double rho = a.q[1][k] + a.q[0][k];
        a.rho[k] = rho;
        if (a.f) a.f[k] = rhs_node(rho, i, j, a, phirx);
    }
}

__global__ void k_rhs(FinalizeArgs a) {
    pgb_pdl_entry();
    const int G = a.nx * a.ny;
    const double phirx = a.phi_tab[a.ds->tf - a.ds->t_base];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < G; k += gridDim.x * blockDim.x) {
        int j = k / a.nx, i = k - j * a.nx;
        a.f[k] = rhs_node(a.rho[k], i, j, a, phirx);
    }
}

/* ------------------------------------------------------- E field */
/* fields::grid_electric_field (fields.cpp:230-268) in the stride-nx layout
 * of an (nx+1)*(ny+1) buffer; also writes the FP32 {Ex,Ey} copy read by
 * the gather.                                                           */
__device__ __forceinline__ double ex_interior(const double* phi, int nx, int ny, int j, int i, double twoDX) {
    if (j < 1 || j > ny - 2 || i < 1 || i > nx - 2) return 0.0;
    return (phi[j * nx + i - 1] - phi[j * nx + i + 1]) / twoDX;
}
__device__ __forceinline__ double ey_interior(const double* phi, int nx, int ny, int j, int i, double twoDX) {
    if (j < 1 || j > ny - 2 || i < 1 || i > nx - 2) return 0.0;
    return (phi[(j - 1) * nx + i] - phi[(j + 1) * nx + i]) / twoDX;
}
__global__ void k_efield(const double* phi, double* Ex, double* Ey, float2* exy, int nx, int ny, double twoDX,
                         DevState* ds, int advance) {
    pgb_pdl_entry();
    /* the last kernel of a field solve moves the field step counter on */
    if (advance && blockIdx.x == 0 && threadIdx.x == 0) ds->tf += 1;
    const int GE = (nx + 1) * (ny + 1);
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < GE; k += gridDim.x * blockDim.x) {
        double ex = 0.0, ey = 0.0;
        if (k < nx * ny) {
            int j = k / nx, i = k - j * nx;
            if (i == 0) ex = 2.0 * ex_interior(phi, nx, ny, j, 1, twoDX) - ex_interior(phi, nx, ny, j, 2, twoDX);
            else if (i == nx - 1) ex = 2.0 * ex_interior(phi, nx, ny, j, nx - 2, twoDX) - ex_interior(phi, nx, ny, j, nx - 3, twoDX);
            else ex = ex_interior(phi, nx, ny, j, i, twoDX);
            if (j == 0) ey = 2.0 * ey_interior(phi, nx, ny, 1, i, twoDX) - ey_interior(phi, nx, ny, 2, i, twoDX);
            else if (j == ny - 1) ey = 2.0 * ey_interior(phi, nx, ny, ny - 2, i, twoDX) - ey_interior(phi, nx, ny, ny - 3, i, twoDX);
            else ey = ey_interior(phi, nx, ny, j, i, twoDX);
        }
        Ex[k] = ex;
        Ey[k] = ey;
        exy[k] = make_float2((float)ex, (float)ey);
    }
}

__global__ void k_walls(double* phi, int nx, int ny, double phi0x, const double* phi_tab, const DevState* ds,
                        double phi0y, double phily) {
    pgb_pdl_entry();
    const double phirx = phi_tab[ds->tf - ds->t_base];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nx * ny; k += gridDim.x * blockDim.x) {
        int j = k / nx, i = k - j * nx;
        /* fields.cpp:209-219: columns first, then rows overwrite the corners */
        if (j == 0) phi[k] = phi0y;
        else if (j == ny - 1) phi[k] = phily;
        else if (i == 0) phi[k] = phi0x;
        else if (i == nx - 1) phi[k] = phirx;
    }
}

/* ====================================================== host side */
static FinalizeArgs fin_args(pgb_run* r, int mask, bool rhs) {
    FinalizeArgs a;
    a.acc[0] = r->qacc[0]; a.acc[1] = r->qacc[1];
    a.q[0] = r->q[0]; a.q[1] = r->q[1];
    a.rho = r->rho; a.f = rhs ? r->mg_f[r->ng - 1] : nullptr;
    a.nx = r->nx; a.ny = r->ny;
    a.qcdxdy[0] = r->sp[0].qc / (r->dx * r->dy);
    a.qcdxdy[1] = r->sp[1].qc / (r->dx * r->dy);
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

/* One defect-correction update: u' = u + e in FP64 (u' = e on the first
 * pass, when u is null), written to a second buffer so that neighbours
 * read the old values, and the FP64 defect d = f - L u' of the interior
 * (zero on the walls) stored as FP32 for the next FP32 correction.  The
 * walls of u, e and so u' are 0.                                         */
__global__ void k_dc_update(const double* __restrict__ u, const float* __restrict__ e, double* __restrict__ uout,
                            const double* __restrict__ f, float* __restrict__ d, int n, double h2i) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n * n; k += gridDim.x * blockDim.x) {
        int i = k / n, j = k - i * n;
        auto U = [&](int q) { return u ? u[q] + (double)e[q] : (double)e[q]; };
        double c = U(k), v = 0.0;
        if (i > 0 && j > 0 && i < n - 1 && j < n - 1)
            v = f[k] - h2i * (U(k + n) + U(k - n) + U(k + 1) + U(k - 1) - 4.0 * c);
        uout[k] = c;
        d[k] = (float)v;
    }
}
/* the last correction: phi = u + e in FP64 (the walls are set after) */
__global__ void k_dc_final(double* __restrict__ phi, const double* __restrict__ u, const float* __restrict__ e,
                           int count) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x)
        phi[k] = u[k] + (double)e[k];
}
/* DST_DC: the FP32 right-hand side of the charge alone, -rho/EPSILON on
 * the interior (the walls' terms are in the wall solutions)             */
__global__ void k_rho32(float* __restrict__ f32, const double* __restrict__ rho, int n, double coef) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n * n; k += gridDim.x * blockDim.x) {
        int i = k / n, j = k - i * n;
        f32[k] = (i > 0 && j > 0 && i < n - 1 && j < n - 1) ? (float)(-coef * rho[k]) : 0.0f;
    }
}
/* DST_DC's first update: u = wc + phi_right(t) * wr + e (the walls' FP64
 * solutions and the FP32 solve of the charge term), and the FP64 defect
 * d = f - L u of the full right-hand side, as k_dc_update            */
__global__ void k_dc_first(const double* __restrict__ wc, const double* __restrict__ wr, const double* phi_tab,
                           const DevState* ds, const float* __restrict__ e, double* __restrict__ uout,
                           const double* __restrict__ f, float* __restrict__ d, int n, double h2i) {
    pgb_pdl_entry();
    const double phirx = phi_tab[ds->tf - ds->t_base];
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n * n; k += gridDim.x * blockDim.x) {
        int i = k / n, j = k - i * n;
        auto U = [&](int q) { return (wc[q] + phirx * wr[q]) + (double)e[q]; };
        double c = U(k), v = 0.0;
        if (i > 0 && j > 0 && i < n - 1 && j < n - 1)
            v = f[k] - h2i * (U(k + n) + U(k - n) + U(k + 1) + U(k - 1) - 4.0 * c);
        uout[k] = c;
        d[k] = (float)v;
    }
}
/* the walls' terms of the right-hand side alone (rhs_node at rho = 0) */
__global__ void k_wall_rhs(FinalizeArgs a, double phirx) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < a.nx * a.ny; k += gridDim.x * blockDim.x) {
        int j = k / a.nx, i = k - j * a.nx;
        a.f[k] = rhs_node(0.0, i, j, a, phirx);
    }
}
__global__ void k_to32(float* d, const double* s, int count) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) d[k] = (float)s[k];
}
__global__ void k_to64(double* d, const float* s, int count) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) d[k] = (double)s[k];
}

/* FP64 defect correction around the FP32 sine-transform solve of L u = f64
 * (zero walls), `passes` solves in all; the result goes to out (FP64).
 * lift: the first approximation is the walls' solution wc + phi_right(t) wr
 * plus the FP32 solve of the charge term alone, which keeps the walls'
 * terms (-phi/(DX DY) next to a wall, a thousand times the charge term at
 * 1 V) out of the FP32 transform, whose rounding they would otherwise
 * spread over every mode; each pass then divides the error by about 1e6
 * instead of about 300.  Otherwise the first solve is of f64 itself.  */
static int dst_dc(pgb_run* r, const double* f64, double* out, int passes, bool lift) {
    const int top = r->ng - 1, n = r->nx, G = n * n, gb = blocks_for(G);
    const double h = r->p.xlength / (n - 1), h2i = 1.0 / (h * h);
    float* const f32 = r->mg32_f[top];   /* right-hand side, then each defect */
    float* const e32 = r->mg32_u[top];   /* each FP32 solve                   */
    if (lift) PGB_CK(r, pgb_launch_pdl(k_rho32, dim3(gb), dim3(256), 0, r->stream, f32, (const double*)r->rho, n,
                                       1.0 / 8.854e-12));
    else PGB_CK(r, pgb_launch_pdl(k_to32, dim3(gb), dim3(256), 0, r->stream, f32, f64, G));
    r->launches++;
    if (pgb_dst_solve(r, f32, e32)) return PGB_ERR_CUDA;
    if (passes <= 1 && !lift) {
        PGB_CK(r, pgb_launch_pdl(k_to64, dim3(gb), dim3(256), 0, r->stream, out, (const float*)e32, G));
        r->launches++;
        return 0;
    }
    double* ua = nullptr;   /* FP64 solution so far */
    double* ub = passes <= 1 ? out : r->dc_u;
    if (lift) {
        PGB_CK(r, pgb_launch_pdl(k_dc_first, dim3(gb), dim3(256), 0, r->stream, (const double*)r->dst_wc,
                                 (const double*)r->dst_wr, (const double*)r->phi_tab, (const DevState*)r->ds,
                                 (const float*)e32, ub, f64, f32, n, h2i));
        r->launches++;
        if (passes <= 1) return 0;
        ua = ub;
        ub = r->dc_u2;
        if (pgb_dst_solve(r, f32, e32)) return PGB_ERR_CUDA;
    }
    for (int it = lift ? 2 : 1; it < passes; ++it) {
        PGB_CK(r, pgb_launch_pdl(k_dc_update, dim3(gb), dim3(256), 0, r->stream, (const double*)ua, (const float*)e32,
                                 ub, f64, f32, n, h2i));
        r->launches++;
        ua = ub;
        ub = (ub == r->dc_u) ? r->dc_u2 : r->dc_u;
        if (pgb_dst_solve(r, f32, e32)) return PGB_ERR_CUDA;
    }
    PGB_CK(r, pgb_launch_pdl(k_dc_final, dim3(gb), dim3(256), 0, r->stream, out, (const double*)ua, (const float*)e32, G));
    r->launches++;
    return 0;
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
    for (int w = 0; w < 2; ++w) {
        FinalizeArgs a = fin_args(r, 0, true);
        a.f = f64;
        if (w == 1) a.phi0x = a.phi0y = a.phily = 0.0;
        PGB_CK(r, pgb_launch_pdl(k_wall_rhs, dim3(blocks_for((long long)G)), dim3(256), 0, r->stream, a,
                                 w == 1 ? 1.0 : 0.0));
        if (dst_dc(r, f64, w == 0 ? r->dst_wc : r->dst_wr, 8, false)) return PGB_ERR_CUDA;
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
int pgb_poisson_solve(pgb_run* r) {
    const int top = r->ng - 1, n = r->nx;
    const int G = n * n;
    const int gb = blocks_for(G);
    if (r->p.poisson_mode == PGB_POISSON_FMG_REF) {
        if (pgb_mg_fmg64(r)) return PGB_ERR_CUDA;
        PGB_CK(r, cudaMemcpyAsync(r->phi, r->mg_u[top], sizeof(double) * G, cudaMemcpyDeviceToDevice, r->stream));
    } else if (r->p.poisson_mode == PGB_POISSON_DST_DC) {
        if (!pgb_dst_ok(r)) return PGB_ERR_CUDA;
        if (dst_dc(r, r->mg_f[top], r->phi, r->p.dc_max_iters > 1 ? r->p.dc_max_iters : 1, true)) return PGB_ERR_CUDA;
    } else {
        PGB_CK(r, pgb_launch_pdl(k_to32, dim3(gb), dim3(256), 0, r->stream, r->mg32_f[top], (const double*)r->mg_f[top], G));
        r->launches++;
        if (pgb_mg_fmg32(r)) return PGB_ERR_CUDA;
        const float* e = r->mg32_u[top];   /* the FMG pass's result        */
        const int passes = r->p.poisson_mode == PGB_POISSON_FP32_DC && r->p.dc_max_iters > 1 ? r->p.dc_max_iters : 1;
        if (passes == 1) {
            PGB_CK(r, pgb_launch_pdl(k_to64, dim3(gb), dim3(256), 0, r->stream, r->phi, e, G));
            r->launches++;
        } else {
            const double h = r->p.xlength / (n - 1), h2i = 1.0 / (h * h);
            double* ua = nullptr;        /* FP64 solution so far (null: 0) */
            double* ub = r->dc_u;
            for (int it = 1; it < passes; ++it) {
                /* the defect goes to the level's residual array, its V-cycle
                 * from 0 to the level's correction array                 */
                PGB_CK(r, pgb_launch_pdl(k_dc_update, dim3(gb), dim3(256), 0, r->stream, (const double*)ua, e, ub,
                                         (const double*)r->mg_f[top], r->mg32_r[top], n, h2i));
                r->launches++;
                ua = ub;
                ub = (ub == r->dc_u) ? r->dc_u2 : r->dc_u;
                if (pgb_mg_vcycle32(r)) return PGB_ERR_CUDA;
                e = r->mg32_v[top];
            }
            PGB_CK(r, pgb_launch_pdl(k_dc_final, dim3(gb), dim3(256), 0, r->stream, r->phi, (const double*)ua, e, G));
            r->launches++;
        }
    }
    PGB_CK(r, pgb_launch_pdl(k_walls, dim3(blocks_for((long long)r->nx * r->ny)), dim3(256), 0, r->stream, r->phi, r->nx, r->ny, r->p.phi_left, r->phi_tab,
                                                                         r->ds, r->p.phi_bottom, r->p.phi_top));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_efield(pgb_run* r, int advance) {
    int GE = (r->nx + 1) * (r->ny + 1);
    PGB_CK(r, pgb_launch_pdl(k_efield, dim3(blocks_for(GE)), dim3(256), 0, r->stream, r->phi, r->ex, r->ey, r->exy, r->nx, r->ny, 2.0 * r->dx, r->ds, advance));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}


