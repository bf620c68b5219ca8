/*
 * The charge deposit of particles in any order (particle::collect_charge,
 * particle.cpp:663-858, pic.cl:22-52) through a window of the grid in
 * shared memory: the grid itself where it is small, else the bounding box
 * of the particles in work, which is small when they come binned, as a
 * sorted run holds and dumps them.
 *
 * A particle adds to four nodes.  As 64-bit atomics at L2 those adds bound
 * the deposit wherever many particles share a node; in the window they are
 * 32-bit shared-memory atomics (native, 64-bit ones are not), and a node
 * goes to L2 once per flush.  A window sum that wraps adds 2^32 to the
 * node's total at once, so a window takes any number of particles.  Both
 * paths add the same integers, round(a w 2^19), so the grid does not depend
 * on the path.
 */
#pragma once
#include "pgb_internal.h"
#include "pgb_physics.cuh"

#define DEP_THREADS 512
#define DEP_ITEMS 4                             /* particles per thread and round  */
#define DEP_CHUNK (DEP_THREADS * DEP_ITEMS)
#define DEP_NODES 16900                         /* window words: a 129 x 129 grid fits */
#define DEP_MARGIN 4                            /* cells added around a bounding box */
#define DEP_SMEM (DEP_NODES * sizeof(unsigned int))
#define DEP_BLOCKS_PER_SM 3

/* Windows pay for their zeroing, their flush and fewer blocks in flight from
 * 16 particles a node (8192 in all): straight (deposit_pairs) / windows, the
 * kernel alone, 17^2 nodes, 5000 particles 4.0 / 5.5 us, 20 K 9.6 / 5.6;
 * 65^2, 50 K 4.8 / 7.2, 131 K 7.5 / 7.4, 1 M 34 / 12; 129^2, 300 K 9.8 / 11.6,
 * 1 M 27 / 18.  On larger grids they pay if the particles come binned, which
 * the caller of a large deposit mostly has them: records, 257^2, 1 M 23 / 29
 * in random order and 27 / 21 in bins, 6 M 119 / 163 and 226 / 104; 513^2,
 * 2.5 M 48 / 68 and 55 / 58, 6 M 102 / 159 and 158 / 113.                 */
inline bool deposit_through_windows(int64_t n, int64_t nodes) { return n >= 8192 && n >= 16 * nodes; }

struct DepWindow {
    unsigned int* w;
    int ox, oy, nx, ny;   /* first node, nodes a row, rows */
    bool live;
};

/* round(v) to nearest even for 0 <= v < 2^22, as __float2int_rn: adding
 * 1.5 * 2^23 leaves v's integer part in the low mantissa bits, rounded by
 * the addition itself (1.5 * 2^23 is even, so ties go the same way)      */
__device__ __forceinline__ unsigned int round_small(float v) {
    return (unsigned int)__float_as_int(__fadd_rn(v, 12582912.0f)) - 0x4b400000u;
}

__device__ __forceinline__ void dep_zero(const DepWindow& W) {
    for (int k = threadIdx.x; k < W.nx * W.ny; k += DEP_THREADS) W.w[k] = 0u;
    __syncthreads();
}
/* the window's sums to the grid; a warp per row, a lane per node */
__device__ __forceinline__ void dep_flush(const DepWindow& W, unsigned long long* acc, int nx) {
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int r = threadIdx.x >> 5; r < W.ny; r += DEP_THREADS / 32) {
        unsigned long long* const row = acc + (long long)(W.oy + r) * nx + W.ox;
        for (int c = lane; c < W.nx; c += 32) {
            const unsigned int v = W.w[r * W.nx + c];
            if (v) atomicAdd(row + c, (unsigned long long)v);
        }
    }
    __syncthreads();
}
__device__ __forceinline__ void dep_add(const DepWindow& W, unsigned long long* acc, int nx, int k, float a, float wS) {
    const unsigned int v = round_small(__fmul_rn(a, wS));
    const unsigned int old = atomicAdd(&W.w[k], v);
    if (old + v < old) {   /* wrapped */
        const int r = k / W.nx;
        atomicAdd(acc + (long long)(W.oy + r) * nx + W.ox + (k - r * W.nx), 1ull << 32);
    }
}

/* The deposits of a warp's particles (`ok` ones) straight to the grid, two
 * lanes to a particle: a lane adds to one column's two nodes of its own
 * particle and of its neighbour's, so that the two nodes of a row, which
 * mostly share a sector, go to L2 as one request (all 32 lanes call it).
 * With four adds of its own per lane, unsorted argon runs took per step:
 * 257^2 nodes, 300 K particles a species 55 us, now 49, 4 M 308, now 243;
 * 513^2, 8 M 550, now 466.                                               */
__device__ __forceinline__ void deposit_pairs(unsigned long long* qacc, int nx, int ps, bool ok, float xs, float ys,
                                              float w) {
    if (ok && !(w >= 0.0f && w < 1.99f)) {
        deposit_cell(qacc, nx, ps, xs, ys, w);
        ok = false;
    }
    const bool odd = threadIdx.x & 1;
    const float wj = pfrac(xs, ps), wk = pfrac(ys, ps), wS = w * PGB_FIX_SCALE_F;
    const unsigned v0 = round_small(__fmul_rn((1.0f - wj) * (1.0f - wk), wS)), v1 = round_small(__fmul_rn(wj * (1.0f - wk), wS));
    const unsigned v2 = round_small(__fmul_rn(wk * (1.0f - wj), wS)), v3 = round_small(__fmul_rn(wj * wk, wS));
    const int k = ok ? (pbits(ys) >> ps) * nx + (pbits(xs) >> ps) : -1;
    const int ko = __shfl_xor_sync(0xffffffffu, k, 1);
    const unsigned a = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1), b = __shfl_xor_sync(0xffffffffu, odd ? v2 : v3, 1);
    /* even lanes take the left column, odd lanes the right one */
    unsigned long long* const q = qacc + (odd ? 1 : 0);
    const int ke = odd ? ko : k, kd = odd ? k : ko;   /* the even and the odd lane's particle */
    if (ke >= 0) {
        atomicAdd(q + ke, (unsigned long long)(odd ? a : v0));
        atomicAdd(q + ke + nx, (unsigned long long)(odd ? b : v2));
    }
    if (kd >= 0) {
        atomicAdd(q + kd, (unsigned long long)(odd ? v1 : a));
        atomicAdd(q + kd + nx, (unsigned long long)(odd ? v3 : b));
    }
}

/* All particles i in [0, n) of src, which returns a particle's fixed-point
 * position lanes and weight (a dead one where it has none).  Blocks of
 * DEP_THREADS; a block takes a run of consecutive particles.             */
template <class Src>
__device__ __forceinline__ void deposit_windows(const Src& src, long long n, int nx, int ny, int ps,
                                                unsigned long long* acc) {
    extern __shared__ __align__(16) unsigned int s_dep[];
    __shared__ int s_box[4][DEP_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const bool whole = nx * ny <= DEP_NODES;
    DepWindow W{s_dep, 0, 0, nx, ny, whole};
    const long long chunks = (n + DEP_CHUNK - 1) / DEP_CHUNK, per = (chunks + gridDim.x - 1) / gridDim.x;
    const long long c0 = per * blockIdx.x, c1 = c0 + per < chunks ? c0 + per : chunks;
    if (c0 >= c1) return;
    if (whole) dep_zero(W);
    for (long long c = c0; c < c1; ++c) {
        float x[DEP_ITEMS], y[DEP_ITEMS], w[DEP_ITEMS];
#pragma unroll
        for (int q = 0; q < DEP_ITEMS; ++q) {
            const long long i = c * DEP_CHUNK + q * DEP_THREADS + threadIdx.x;
            x[q] = y[q] = pos_dead();
            w[q] = 0.0f;
            if (i < n) src(i, x[q], y[q], w[q]);
        }
        bool ok[DEP_ITEMS];
        int lo_x = 1 << 30, lo_y = 1 << 30, hi_x = -1, hi_y = -1;
#pragma unroll
        for (int q = 0; q < DEP_ITEMS; ++q) {
            ok[q] = deposit_ok(x[q], y[q], nx, ny, ps);
            if (ok[q] && !(w[q] >= 0.0f && w[q] < 1.99f)) {   /* a sum of others may not fit the window's word */
                deposit_cell(acc, nx, ps, x[q], y[q], w[q]);
                ok[q] = false;
            }
            if (ok[q]) {
                const int j = pbits(x[q]) >> ps, k = pbits(y[q]) >> ps;
                lo_x = min(lo_x, j); hi_x = max(hi_x, j);
                lo_y = min(lo_y, k); hi_y = max(hi_y, k);
            }
        }
        if (!whole) {
            lo_x = __reduce_min_sync(0xffffffffu, lo_x);
            lo_y = __reduce_min_sync(0xffffffffu, lo_y);
            hi_x = __reduce_max_sync(0xffffffffu, hi_x);
            hi_y = __reduce_max_sync(0xffffffffu, hi_y);
            if (lane == 0) {
                s_box[0][warp] = lo_x; s_box[1][warp] = lo_y;
                s_box[2][warp] = hi_x; s_box[3][warp] = hi_y;
            }
            __syncthreads();
#pragma unroll
            for (int v = 0; v < DEP_THREADS / 32; ++v) {
                lo_x = min(lo_x, s_box[0][v]); lo_y = min(lo_y, s_box[1][v]);
                hi_x = max(hi_x, s_box[2][v]); hi_y = max(hi_y, s_box[3][v]);
            }
            __syncthreads();
            if (hi_x < 0) continue;   /* nothing to deposit in this round */
            const bool inside = W.live && lo_x >= W.ox && lo_y >= W.oy && hi_x + 1 < W.ox + W.nx && hi_y + 1 < W.oy + W.ny;
            if (!inside) {
                if (W.live) dep_flush(W, acc, nx);
                /* the box with a margin where that fits, so that the next
                 * rounds of the same bin stay inside                      */
                for (int m = DEP_MARGIN; m >= 0; m -= DEP_MARGIN) {
                    W.ox = max(lo_x - m, 0);
                    W.oy = max(lo_y - m, 0);
                    W.nx = min(hi_x + 1 + m, nx - 1) - W.ox + 1;
                    W.ny = min(hi_y + 1 + m, ny - 1) - W.oy + 1;
                    W.live = W.nx * W.ny <= DEP_NODES;
                    if (W.live) break;
                }
                if (W.live) dep_zero(W);
            }
        }
        if (!W.live) {
#pragma unroll
            for (int q = 0; q < DEP_ITEMS; ++q) deposit_pairs(acc, nx, ps, ok[q], x[q], y[q], w[q]);
            continue;
        }
#pragma unroll
        for (int q = 0; q < DEP_ITEMS; ++q) {
            if (!ok[q]) continue;
            const int k = ((pbits(y[q]) >> ps) - W.oy) * W.nx + (pbits(x[q]) >> ps) - W.ox;
            const float wj = pfrac(x[q], ps), wk = pfrac(y[q], ps), wS = w[q] * PGB_FIX_SCALE_F;
            dep_add(W, acc, nx, k, (1.0f - wj) * (1.0f - wk), wS);
            dep_add(W, acc, nx, k + 1, wj * (1.0f - wk), wS);
            dep_add(W, acc, nx, k + W.nx, wk * (1.0f - wj), wS);
            dep_add(W, acc, nx, k + W.nx + 1, wj * wk, wS);
        }
    }
    if (W.live) dep_flush(W, acc, nx);
}
