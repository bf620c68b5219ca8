/*
 * Headless viewer plots: the plots of the reference's OpenGL viewer
 * (graphics.cpp:245-607) rasterised by CUDA into an RGB8 image owned by the
 * run.  The GL window itself needs a graphics stack; the plots are plain
 * rasterisation and need none.
 *
 * Particle plots (two order-independent passes over the particle arrays):
 *   - a particle is plotted when it is live, in the sample (a hash of its
 *     id, see rd_keep) and strictly inside the domain in FP32 cell units
 *     (the |x| < boxLength/2 test of graphics.cpp:432-436, 593-595);
 *   - vx-vy: k_rd_vmax takes the largest |vx| and |vy| of those particles
 *     (atomicMax on the float bits, exact), k_rd_points truncates it to an
 *     int, at least 1 (graphics.cpp:421-452), and plots the particles with
 *     |vx|, |vy| below it (graphics.cpp:499-503);
 *   - a point is 2 x 2 pixels (glPointSize(2), graphics.cpp:483).  Points
 *     set bits of a one-bit-per-pixel layer per species (see rd_mark);
 *     k_rd_resolve turns the layers into colours, ions over electrons.
 *   - Blocks take 4096-particle tiles in a scrambled order (tile t * P mod
 *     ntiles, P a prime above any tile count): spatially sorted particles
 *     would otherwise put the blocks in flight on the same few words.
 * Field plots (k_rd_field, one thread per pixel): the pixel's grid
 * coordinate picks a cell; the cell's quad is inset by a tenth of a cell,
 * and its colour is the ramp of drawField (graphics.cpp:303-356) applied to
 * |mean of the four corners / max|.  The maximum comes from k_rd_fmax, an
 * order-independent max over the field (NaN values ignored), the corners'
 * values from k_rd_nodes.
 *
 * The unit is compiled with --fmad=false so that every pixel and colour
 * equals the oracle's C restatement of the same rules bit for bit.
 */
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>
#include <algorithm>
#include "pgb_internal.h"
#include "pgb_physics.cuh"

namespace {

struct Rgb { unsigned char r, g, b; };

/* colour byte of a [0,1] component */
__device__ __forceinline__ unsigned char rd_byte(float c) {
    float v = c * 255.0f + 0.5f;
    v = v < 0.0f ? 0.0f : (v > 255.0f ? 255.0f : v);
    return (unsigned char)(int)v;
}

/* lowbias32 integer hash (C. Wellons, hash-prospector) of id and seed */
__device__ __forceinline__ uint32_t rd_hash(uint32_t id, uint32_t seed) {
    uint32_t x = id ^ (seed * 0x9E3779B9u);
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

/* the sample: all particles when max_points <= 0 or n <= max_points, else
 * those with hash < max_points/n of the 32-bit range                     */
struct RdSample {
    bool all;
    unsigned long long thresh;
    __device__ __forceinline__ RdSample(int max_points, long long nlive)
        : all(max_points <= 0 || nlive <= max_points),
          thresh(all ? 0ull : (unsigned long long)((double)max_points / (double)nlive * 4294967296.0)) {}
};

struct PointArgs {
    const float4* xv;
    const unsigned int* id;
    const DevState* ds;
    int s, nx, ny, ps, width, height, max_points, phase;
    uint32_t seed;
    const unsigned int* vmax;   /* phase: bits of max |vx|, |vy| */
    unsigned int* vmax_out;     /* k_rd_vmax */
    unsigned int* layer;        /* one bit per pixel */
    int words;                  /* of the layer */
    int shared;                 /* the layer fits in shared memory */
};

#define RD_TILE 4096
#define RD_THREADS 1024
#define RD_SCRAMBLE 2147483647ull   /* 2^31-1, prime and above any tile count (at most 2^21):
                                      t -> t * P mod ntiles is a permutation */

__device__ __forceinline__ long long rd_tile(long long t, long long ntiles) {
    return (long long)(((unsigned long long)t * RD_SCRAMBLE) % (unsigned long long)ntiles);
}

/* p.x, p.y: the position in FP32 cells (NaN for a NaN position) */
__device__ __forceinline__ bool rd_candidate(const PointArgs& a, float4& p) {
    if (is_dead(p.x)) return false;
    p.x = pos_cellsf(p.x, a.ps);
    p.y = pos_cellsf(p.y, a.ps);
    return p.x > 0.0f && p.x < (float)(a.nx - 1) && p.y > 0.0f && p.y < (float)(a.ny - 1);
}
/* f(particle) for the sampled slots of the block's tiles; a thread's items
 * load together.  A sample is decided by the ids alone (4 B a slot), and
 * only its particles are read: 5000 of 2 x 16 M drawn at 1024^2 pixels took
 * 240 us when the ids were read after the positions, now 141 (all 253).  */
template <class F>
__device__ __forceinline__ void rd_particles(const PointArgs& a, long long n, long long nlive, F f) {
    const long long ntiles = (n + RD_TILE - 1) / RD_TILE;
    const RdSample smp(a.max_points, nlive);
    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long base = rd_tile(t, ntiles) * RD_TILE;
        float4 p[RD_TILE / RD_THREADS];
        unsigned int id[RD_TILE / RD_THREADS];
        if (!smp.all) {
#pragma unroll
            for (int q = 0; q < RD_TILE / RD_THREADS; ++q) {
                const long long i = base + q * RD_THREADS + threadIdx.x;
                id[q] = i < n ? a.id[i] : 0u;
            }
        }
#pragma unroll
        for (int q = 0; q < RD_TILE / RD_THREADS; ++q) {
            const long long i = base + q * RD_THREADS + threadIdx.x;
            const bool keep = i < n && (smp.all || (unsigned long long)rd_hash(id[q], a.seed) < smp.thresh);
            p[q] = keep ? a.xv[i] : make_float4(pos_dead(), 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int q = 0; q < RD_TILE / RD_THREADS; ++q) f(p[q]);
    }
}

__global__ void __launch_bounds__(RD_THREADS) k_rd_vmax(PointArgs a) {
    const long long n = a.ds->n[a.s], nlive = n - a.ds->dead[a.s];
    unsigned int mx = 0u, my = 0u;
    rd_particles(a, n, nlive, [&](float4 p) {
        if (!rd_candidate(a, p)) return;
        const float ax = fabsf(p.z), ay = fabsf(p.w);
        if (ax == ax) mx = max(mx, __float_as_uint(ax));   /* non-negative floats order as their bits */
        if (ay == ay) my = max(my, __float_as_uint(ay));
    });
    mx = __reduce_max_sync(0xffffffffu, mx);
    my = __reduce_max_sync(0xffffffffu, my);
    if ((threadIdx.x & 31) == 0) {
        if (mx) atomicMax(&a.vmax_out[0], mx);
        if (my) atomicMax(&a.vmax_out[1], my);
    }
}

/* (int) of a non-negative float, at least 1 (int maxVx, graphics.cpp:421-452) */
__device__ __forceinline__ int rd_vscale(unsigned int bits) {
    float v = __uint_as_float(bits);
    int m = v < 2147483520.0f ? (int)v : 2147483647;
    return m < 1 ? 1 : m;
}

/* The pixels that points cover are bits: a block marks them in its own copy
 * of the layer in shared memory (an image of 1.6 M pixels fits) and adds
 * that to the layer at its end; a larger image is marked in the layer
 * itself.  Marks are only set, in any order, so the image does not depend on
 * it; a bit already seen set needs no atomic.  With a byte per pixel in
 * global memory, read and stored by every point, the X-Y frame of 3 M
 * particles at 768^2 took 2 x 160 us.                                     */
__device__ __forceinline__ void rd_mark(unsigned int* w, unsigned int m) {
    if ((*(volatile unsigned int*)w & m) != m) atomicOr(w, m);
}
/* a 2 x 2 point with its lower left pixel at (px, py) */
__device__ __forceinline__ void rd_splat(const PointArgs& a, unsigned int* layer, int px, int py) {
    const int cols = px + 1 < a.width ? 2 : 1;
    for (int dy = 0; dy < 2; ++dy) {
        const int y = py - dy;
        if (y < 0) continue;
        const unsigned int k = (unsigned int)y * a.width + px, b = k & 31;
        const unsigned int m = cols == 2 ? 3u : 1u;
        rd_mark(layer + (k >> 5), m << b);
        if (cols == 2 && b == 31) rd_mark(layer + (k >> 5) + 1, 1u);
    }
}

/* layer bits -> colours: c2 over c1 over black; four pixels a thread */
__global__ void k_rd_resolve(const unsigned int* l1, const unsigned int* l2, long long npx, Rgb c1, Rgb c2,
                             unsigned char* img) {
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; 4 * q < npx; q += (long long)gridDim.x * blockDim.x) {
        const long long k = 4 * q;
        const unsigned int b1 = (l1 ? l1[k >> 5] : 0u) >> (k & 31), b2 = (l2 ? l2[k >> 5] : 0u) >> (k & 31);
        unsigned char v[12];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const Rgb c = (b2 >> j) & 1u ? c2 : (b1 >> j) & 1u ? c1 : Rgb{0, 0, 0};
            v[3 * j] = c.r; v[3 * j + 1] = c.g; v[3 * j + 2] = c.b;
        }
        if (k + 4 <= npx) {
            unsigned int* const o = reinterpret_cast<unsigned int*>(img + 3 * k);
#pragma unroll
            for (int j = 0; j < 3; ++j)
                o[j] = v[4 * j] | (unsigned)v[4 * j + 1] << 8 | (unsigned)v[4 * j + 2] << 16 | (unsigned)v[4 * j + 3] << 24;
        } else {
            for (int j = 0; j < 3 * (int)(npx - k); ++j) img[3 * k + j] = v[j];
        }
    }
}

__global__ void __launch_bounds__(RD_THREADS) k_rd_points(PointArgs a) {
    extern __shared__ unsigned int s_layer[];
    const long long n = a.ds->n[a.s], nlive = n - a.ds->dead[a.s];
    int mvx = 1, mvy = 1;
    if (a.phase) {
        mvx = rd_vscale(a.vmax[0]);
        mvy = rd_vscale(a.vmax[1]);
    }
    const float W = (float)a.width, H = (float)a.height;
    unsigned int* const layer = a.shared ? s_layer : a.layer;
    if (a.shared) {
        for (int k = threadIdx.x; k < a.words; k += RD_THREADS) s_layer[k] = 0u;
        __syncthreads();
    }
    rd_particles(a, n, nlive, [&](float4 p) {
        if (!rd_candidate(a, p)) return;
        float fx, fy;
        if (a.phase) {
            if (!(fabsf(p.z) < (float)mvx && fabsf(p.w) < (float)mvy)) return;
            fx = (p.z / (float)mvx + 1.0f) * 0.5f;
            fy = (p.w / (float)mvy + 1.0f) * 0.5f;
        } else {
            fx = p.x / (float)(a.nx - 1);
            fy = p.y / (float)(a.ny - 1);
        }
        int px = (int)(fx * W), py = a.height - 1 - (int)(fy * H);
        px = px < 0 ? 0 : (px > a.width - 1 ? a.width - 1 : px);
        py = py < 0 ? 0 : (py > a.height - 1 ? a.height - 1 : py);
        rd_splat(a, layer, px, py);
    });
    if (a.shared) {
        __syncthreads();
        for (int k = threadIdx.x; k < a.words; k += RD_THREADS) {
            const unsigned int v = s_layer[k];
            if (v && (a.layer[k] & v) != v) atomicOr(a.layer + k, v);
        }
    }
}

/* doubles as ordered 64-bit keys: max of keys = max of values */
__device__ __forceinline__ unsigned long long rd_key(double v) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ __forceinline__ double rd_unkey(unsigned long long k) {
    unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    double v;
    memcpy(&v, &b, sizeof v);
    return v;
}

/* max over src[k] / div (the field the plot shows), NaN ignored */
__global__ void k_rd_fmax(const double* src, double div, int count, unsigned long long* out) {
    unsigned long long m = 0ull;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        double v = src[k] / div;
        if (v == v) m = max(m, rd_key(v));
    }
    for (int d = 16; d; d >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, d));
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

/* the colour ramp of drawField (graphics.cpp:303-356): red, orange,
 * yellow, green, blue, purple; band b mixes colours b and b+1           */
__constant__ float c_ramp[6][3] = {{1.0f, 0.0f, 0.0f}, {1.0f, 0.396f, 0.0f}, {1.0f, 1.0f, 0.0f},
                                   {0.0f, 1.0f, 0.0f}, {0.0f, 0.0f, 1.0f}, {0.396f, 0.0f, 1.0f}};

__device__ __forceinline__ void rd_ramp(float zAv, float (&c)[3]) {
    const float rd = 0.2f;
    float alpha = zAv < 1.0f ? zAv : 1.0f;
    int b;
    if (zAv < rd) {
        alpha /= rd; b = 0;
    } else if ((double)zAv < 2.0 * (double)rd) {
        alpha = (alpha - rd) / rd; b = 1;
    } else if ((double)zAv < 3.0 * (double)rd) {
        alpha = (float)(((double)alpha - 2.0 * (double)rd) / (double)rd); b = 2;
    } else if ((double)zAv < 4.0 * (double)rd) {
        alpha = (float)(((double)alpha - 3.0 * (double)rd) / (double)rd); b = 3;
    } else {
        alpha = (float)(((double)alpha - 4.0 * (double)rd) / (double)rd); b = 4;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) c[k] = c_ramp[b][k] * (1.0f - alpha) + c_ramp[b + 1][k] * alpha;   /* glm::mix */
}

/* the plotted value of each node, (float)(src / div / max): once per node,
 * not four times per pixel (FP64 divisions; 105 us of a 768^2 frame)       */
__global__ void k_rd_nodes(const double* src, double div, int count, const unsigned long long* fmax_key, float* z) {
    double fmax = fabs(rd_unkey(*fmax_key));
    if (*fmax_key == 0ull || !(fmax >= 1.0)) fmax = 1.0;   /* if (fieldMax < 1.0) fieldMax = 1.0 */
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x)
        z[k] = (float)(src[k] / div / fmax);
}
__global__ void k_rd_field(const float* z, int n, int grid_start, int width, int height, unsigned char* img) {
    const unsigned int npx = (unsigned int)width * (unsigned int)height;
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < npx; k += gridDim.x * blockDim.x) {
        const int py = (int)(k / (unsigned)width), px = (int)(k - (unsigned)py * (unsigned)width);
        const float u = ((float)px + 0.5f) * (float)(n - 1) / (float)width;
        const float v = ((float)(height - 1 - py) + 0.5f) * (float)(n - 1) / (float)height;
        const int i = (int)u, j = (int)v;
        const float fu = u - (float)i, fv = v - (float)j;
        unsigned char* q = img + 3ull * k;
        if (i < grid_start || i >= n - grid_start - 1 || j < grid_start || j >= n - grid_start - 1 || fu < 0.1f ||
            fu > 0.9f || fv < 0.1f || fv > 0.9f) {
            q[0] = q[1] = q[2] = 0;
            continue;
        }
        const float z0 = z[(long long)(j + 1) * n + i], z1 = z[(long long)(j + 1) * n + i + 1];
        const float z2 = z[(long long)j * n + i + 1], z3 = z[(long long)j * n + i];
        const float zAv = (float)fabs((double)(z0 + z1 + z2 + z3) / 4.0);
        float c[3];
        rd_ramp(zAv, c);
        q[0] = rd_byte(c[0]);
        q[1] = rd_byte(c[1]);
        q[2] = rd_byte(c[2]);
    }
}

int rd_fail(pgb_run* r, int code, const char* msg) {
    r->err = msg;
    return code;
}

const Rgb kLime = {142, 255, 29};      /* (0.557, 1.0, 0.114) x 255, rounded */
const Rgb kHotPink = {255, 29, 142};   /* (1.0, 0.114, 0.557) */

}  // namespace

extern "C" int pgb_render(pgb_run* r, int plot, int32_t width, int32_t height, int32_t max_points, uint32_t seed,
                          uint8_t* rgb, int64_t cap) {
    if (!r) return PGB_ERR_ARG;
    if (!rgb || width < 1 || height < 1 || width > 16384 || height > 16384 || plot < 0 || plot > PGB_PLOT_ION_DENSITY)
        return rd_fail(r, PGB_ERR_ARG, "pgb_render: bad argument (plot kind, or a size outside 1..16384)");
    const long long npx = (long long)width * height, bytes = 3 * npx;
    if (cap < bytes) return rd_fail(r, PGB_ERR_ARG, "pgb_render: rgb buffer smaller than width*height*3");
    if (plot <= PGB_PLOT_ION_VX_VY && (r->sp[0].cap == 0 || r->sp[1].cap == 0))
        return rd_fail(r, PGB_ERR_STATE, "pgb_render: load both species first");
    /* the RGB image, then a bit layer per species or the nodes' values */
    const long long words = (npx + 31) / 32 + 1, nodes = (long long)r->nx * r->ny;
    const long long img_bytes = (bytes + 255) & ~255ll;
    const long long need = img_bytes + std::max<long long>(8 * words, 4 * nodes);
    if (need > r->rd_cap) {
        PGB_CK(r, cudaStreamSynchronize(r->stream));
        cudaFree(r->rd_img);
        r->rd_img = nullptr;
        r->rd_cap = 0;
        if (cudaMalloc(&r->rd_img, (size_t)need) != cudaSuccess) {
            cudaGetLastError();
            return rd_fail(r, PGB_ERR_NOMEM, "pgb_render: image allocation failed");
        }
        r->rd_cap = need;
    }
    if (!r->rd_scratch) {
        if (cudaMalloc(&r->rd_scratch, 16) != cudaSuccess) {
            cudaGetLastError();
            return rd_fail(r, PGB_ERR_NOMEM, "pgb_render: scratch allocation failed");
        }
    }
    unsigned char* img = (unsigned char*)r->rd_img;
    PGB_CK(r, cudaMemsetAsync(r->rd_scratch, 0, 16, r->stream));
    if (plot <= PGB_PLOT_ION_VX_VY) {
        unsigned int* const layers = (unsigned int*)(img + img_bytes);
        PGB_CK(r, cudaMemsetAsync(layers, 0, (size_t)(8 * words), r->stream));
        PointArgs a;
        a.ds = r->ds; a.nx = r->nx; a.ny = r->ny; a.ps = r->ps; a.width = width; a.height = height;
        a.max_points = max_points; a.seed = seed;
        a.words = (int)words;
        a.vmax = (const unsigned int*)r->rd_scratch;
        a.vmax_out = (unsigned int*)r->rd_scratch;
        const size_t most = 200 * 1024;
        a.shared = 4 * words <= (long long)most;
        const size_t smem = a.shared ? (size_t)(4 * words) : 0;
        PGB_CK(r, cudaFuncSetAttribute(k_rd_points, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
        const int blocks = r->sms * (smem > 100 * 1024 ? 1 : 2);
        if (plot == PGB_PLOT_PARTICLE_XY) {
            a.phase = 0;
            for (int s = 0; s < 2; ++s) {   /* electrons, then ions on top (graphics.cpp:560-606) */
                a.s = s; a.xv = r->sp[s].xv; a.id = r->sp[s].id;
                a.layer = layers + s * words;
                k_rd_points<<<blocks, RD_THREADS, smem, r->stream>>>(a);
                r->launches++;
            }
        } else {
            const int s = plot == PGB_PLOT_ELECTRON_VX_VY ? 0 : 1;   /* lime / hot pink, graphics.cpp:692, 696 */
            a.phase = 1; a.s = s; a.xv = r->sp[s].xv; a.id = r->sp[s].id;
            a.layer = layers + s * words;
            k_rd_vmax<<<r->sms * 2, RD_THREADS, 0, r->stream>>>(a);
            k_rd_points<<<blocks, RD_THREADS, smem, r->stream>>>(a);
            r->launches += 2;
        }
        const int rb = (int)std::min<long long>((npx + 1023) / 1024, (long long)r->sms * 16);
        k_rd_resolve<<<rb, 256, 0, r->stream>>>(layers, layers + words, npx, kLime, kHotPink, img);
        r->launches++;
    } else {
        const double* src = nullptr;
        double div = 1.0;
        int grid_start = 0;
        const bool averaged = r->gr.on;
        switch (plot) {
            case PGB_PLOT_PHI: src = averaged ? r->gr.f[1] : r->phi; break;
            case PGB_PLOT_EFIELD_X: src = averaged ? r->gr.f[2] : r->ex; break;
            case PGB_PLOT_EFIELD_Y: src = averaged ? r->gr.f[3] : r->ey; break;
            default: {
                const int s = plot == PGB_PLOT_E_DENSITY ? 0 : 1;
                grid_start = 1;   /* graphics.cpp:720, 727 */
                src = averaged ? r->gr.q[s] : r->q[s];
                if (!averaged) div = s == 0 ? -PGB_CHARGE : PGB_CHARGE;   /* q / qc */
            }
        }
        if (averaged) div = (double)r->gr.g.no_graph_steps;
        unsigned long long* key = (unsigned long long*)r->rd_scratch;
        float* const z = (float*)(img + img_bytes);
        const int nb = (int)std::min<long long>((nodes + 255) / 256, (long long)r->sms * 8);
        k_rd_fmax<<<std::min(nb, r->sms * 4), 256, 0, r->stream>>>(src, div, (int)nodes, key);
        k_rd_nodes<<<nb, 256, 0, r->stream>>>(src, div, (int)nodes, key, z);
        const int pb = (int)std::min<long long>((npx + 255) / 256, (long long)r->sms * 16);
        k_rd_field<<<pb, 256, 0, r->stream>>>(z, r->nx, grid_start, width, height, img);
        r->launches += 3;
    }
    PGB_CK(r, cudaGetLastError());
    PGB_CK(r, cudaMemcpyAsync(rgb, img, (size_t)bytes, cudaMemcpyDeviceToHost, r->stream));
    PGB_CK(r, cudaStreamSynchronize(r->stream));
    return 0;
}
