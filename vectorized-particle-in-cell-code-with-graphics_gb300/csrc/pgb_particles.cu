/*
 * Particle kernels: electron-neutral collisions, gather + push + deposit,
 * ordered event lists, injection, ionization products, compaction, load
 * and dump.
 *
 * Reference path: e_collisions::collision (e_collisions.cpp:480-597),
 * particle::get_particle_electric_field + move_particles
 * (particle.cpp:870-1341, pic.cl:56-149), particle::collect_charge
 * (particle.cpp:663-858, pic.cl:22-52), particle::inject_more_particles
 * (particle.cpp:491-510).
 *
 * k_mcc reads each electron (16 B position/velocity, 4 B vz, 4 B id) for
 * the collision test, and handles and writes back the ~5% whose velocity
 * changes; it reads no field, so it runs beside the previous step's field solve.
 * One pass of k_push then reads a particle once (16 B, plus 4 B vz with a
 * magnetic field and 4 B weight), gathers E bilinearly from the FP32 node
 * grid (L2 resident), pushes, deposits the new position into the int64
 * fixed-point charge grid and records wall crossings as per-tile ballot
 * words that keep slot order.  Grids are sized from the SM count and loop over
 * tiles, reading the particle count from device memory, so a step needs
 * no host round trip.
 */
#include <cuda_runtime.h>
#include <math.h>
#include "pgb_internal.h"
#include "pgb_physics.cuh"
#include "pgb_deposit.cuh"
#include "pgb_fp64.cuh"

/* ------------------------------------------------------------ device state */
struct PushArgs {
    float4* xv;
    float* vz;
    float* w;
    const unsigned int* id;
    const float2* exy;
    unsigned long long* qacc;
    DevState* ds;
    int s;
    PushConsts pc;
    CollConsts cc;
    const float* neut;          /* electron-neutral table (FP32), 3 x N */
    const int4* pieces;         /* bin pieces of the last sort              */
    int nbx;                    /* bins per row                             */
    int* tl_out;                /* per-tile outside list              */
    int* tc_out;
    int* tl_ev;                 /* per-tile ionization-event list     */
    int* tc_ev;
};

/* gather (pic.cl:56-92) + push (pic.cl:95-149) of one particle in cell units */
__device__ __forceinline__ void gather_push_one(const PushConsts& pc, const float2* exy, float4& p, float& vz,
                                                bool& moved) {
    moved = false;
    /* jp < nx && x > 0 && kp < ny && y > 0; then the cell is a shift */
    if (pos_open_in(p.x, pc.nx, pc.ps) && pos_open_in(p.y, pc.ny, pc.ps)) {
        const int jp = pbits(p.x) >> pc.ps, kp = pbits(p.y) >> pc.ps;
        float wj = pfrac(p.x, pc.ps), wk = pfrac(p.y, pc.ps);
        float a4 = (1.0f - wj) * (1.0f - wk), a3 = wj * (1.0f - wk);
        float a2 = wk * (1.0f - wj), a1 = wj * wk;
        const float2* e = exy + (long long)kp * pc.nx + jp;
        float2 e0 = __ldg(e), e1 = __ldg(e + 1), e2 = __ldg(e + pc.nx), e3 = __ldg(e + pc.nx + 1);
        float Exp = a4 * e0.x + a3 * e1.x + a2 * e2.x + a1 * e3.x;
        float Eyp = a4 * e0.y + a3 * e1.y + a2 * e2.y + a1 * e3.y;
        float vx = p.z + pc.coef * Exp;
        float vy = p.w + pc.coef * Eyp;
        if (pc.bfield) {
            float vpar = pc.ca * vx + pc.sa * vy;
            float vperp = -pc.sa * vx + pc.ca * vy;
            float vperp_after = vperp * pc.co + pc.so * vz;
            vz = -vperp * pc.so + pc.co * vz;
            vx = pc.ca * vpar - pc.sa * vperp_after;
            vy = pc.sa * vpar + pc.ca * vperp_after;
        }
        vx += pc.coef * Exp;
        vy += pc.coef * Eyp;
        const float dx = pc.dtdx * vx, dy = pc.dtdy * vy;
        /* x and y are below 2^29 + 2^ps here, so a displacement below 2^28
         * needs none of pos_step's limits (a NaN fails the test)          */
        if (fabsf(dx) + fabsf(dy) < 268435456.0f) {
            p.x = plane(pbits(p.x) + __float2int_rn(dx));
            p.y = plane(pbits(p.y) + __float2int_rn(dy));
        } else {
            p.x = pos_step(p.x, dx);
            p.y = pos_step(p.y, dy);
        }
        p.z = vx;
        p.w = vy;
        moved = true;
    }
}

/* electron-neutral collision test (e_collisions.cpp:504-551): both
 * probabilities come from the energy before any event; the decisions are
 * a bit set MCC_SCATTER | MCC_IONIZE.  The scattering continues the EMCC
 * stream after the test's first draw.                                    */
#define MCC_SCATTER 1
#define MCC_IONIZE 2
/* |v|^2 with its roundings spelled out: the collision test and the
 * scatterings must derive the same energy from the same velocity        */
__device__ __forceinline__ float speed2(const float4& p, float vz) {
    return __fmaf_rn(vz, vz, __fmaf_rn(p.w, p.w, __fmul_rn(p.z, p.z)));
}
/* The test in two parts.  mcc_draw: in the domain (0 <= jp < nx,
 * 0 <= kp < ny), |v|^2 and the elastic test's uniform R, the first draw
 * of the electron's EMCC stream; false outside (no event).              */
__device__ __forceinline__ bool mcc_draw(const CollConsts& cc, unsigned int id, unsigned int step, int nx, int ny,
                                         int ps, const float4& p, float vz, float& u2, float& R) {
    if (!(pos_trunc_in(p.x, nx, ps) && pos_trunc_in(p.y, ny, ps))) return false;
    u2 = speed2(p, vz);
    pgb_stream st;
    pgb_stream_init(&st, cc.seed, id, step, PGB_STREAM_EMCC, 0);
    R = pgb_u01f(pgb_stream_u32(&st));
    return true;
}
/* whether mcc_decide can find an event: the elastic bound below with a
 * margin of 1e-5 over its own (about 3e-7 of FP32 rounding, the square
 * root included), written without the square root as u^2 K^2 > 4 R^2
 * (K^2 = cc.el_bound2), or an energy at or above the lowest at which the
 * ionization fit is non-zero (cc.ion_emin).  A false here is a decision
 * of no event that mcc_decide would take too.                           */
__device__ __forceinline__ bool mcc_candidate(const CollConsts& cc, float u2, float R) {
    return (R < 0.5f && u2 * cc.el_bound2 > (2.0f * R) * (2.0f * R)) || cc.e_energy_coef * u2 >= cc.ion_emin;
}
/* the decisions from |v|^2 and R (bit set MCC_SCATTER | MCC_IONIZE) */
__device__ __forceinline__ int mcc_decide(const CollConsts& cc, float u2, float R) {
    float energy = cc.e_energy_coef * u2;
    float u = sqrtf(u2);
    int ev = 0;
    /* P = 1 - exp(-x) is at most 1, so P > 2R cannot hold for R >= 1/2;
     * and P <= x <= u*pcoef*el_max, so with that bound (times 1 + 1e-6,
     * above the FP32 roundings of x and of expm1) at most 2R the event is
     * ruled out: the cross-section and the exponential are needed only
     * for the few electrons left, and every decision is the one the full
     * test would take                                                    */
    if (R < 0.5f && (u * cc.e_pcoef) * cc.el_max * 1.000001f > 2.0f * R) {
        float sel = sigma_el(cc, energy);
        float P = -expm1f(-(u * cc.e_pcoef * sel));
        if (P > 2.0f * R) ev |= MCC_SCATTER;
    }
    /* the ionization test is P = 1 - exp(-x) > 0 (e_collisions.cpp:546-551),
     * which holds exactly when x > 0 (for NaN x neither holds)          */
    float sio = sigma_ion(cc, energy);
    if (u * cc.e_pcoef * sio > 0.0f) ev |= MCC_IONIZE;
    return ev;
}

/* the full ionization of a parent electron (never reached while the
 * reference's energy units make the excess negative): kept out of line so
 * that it does not weigh on the push kernels' registers                  */
__device__ __noinline__ void mcc_ionize_full(const CollConsts& cc, const float* neut, unsigned int id, unsigned int step,
                                             float4& p, float& vz) {
    pgb_stream si;
    pgb_stream_init(&si, cc.seed, id, step, PGB_STREAM_IONIZE, 0);
    /* positions enter only the products; the parent keeps its position */
    IonizeOut o = ionize_f32(&si, neut, cc.n_neutral, cc, 0.0, 0.0, p.z, p.w, vz);
    p.z = (float)o.evx; p.w = (float)o.evy; vz = (float)o.evz;
}

/* e_collisions::ionization's effect on the parent electron, from its
 * velocity after any scattering (e_collisions.cpp:319-443)              */
__device__ __forceinline__ void mcc_ionize(const CollConsts& cc, const float* neut, unsigned int id, unsigned int step,
                                           float4& p, float& vz) {
    if (p.z * p.z + p.w * p.w + vz * vz < cc.ion_vcap * cc.ion_vcap) {
        /* (rm/2)(ve-vn)^2 - THRESHOLD < 0 at this speed for every neutral
         * of the table, so ionize_f32 would return NaN velocities from
         * sqrt of a negative number whatever it draws                   */
        p.z = p.w = vz = __int_as_float(0x7fffffff);
    } else {
        mcc_ionize_full(cc, neut, id, step, p, vz);
    }
}

/* add per-thread event counts (elastic, ionization) with one atomic per
 * warp; the ionizations also to *events, if given                        */
__device__ __forceinline__ void flush_stats(int (&st)[2], long long* stats, long long* events) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        int v = st[k];
        for (int d = 16; d; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
        if ((threadIdx.x & 31) == 0 && v) {
            atomicAdd((unsigned long long*)&stats[ST_ELASTIC + k], (unsigned long long)v);
            if (k == 1 && events) atomicAdd((unsigned long long*)events, (unsigned long long)v);
        }
    }
}

/* A tile's ordered list as bit masks: item k of thread t is slot
 * tile*TILE + k*THREADS + t, so word k*warps + w of the tile (the ballot of
 * warp w's item k) holds its slots in slot order, and the words in order
 * are the tile's list.  The tile's count goes through a shared counter:
 * one barrier per tile, and no scan (k_build_list expands the words).
 * s_cnt: two shared counters, zero at the kernel's start, used by turns
 * (it counts the calls of the block), so that a block's next tile can
 * count while thread 0 reads and clears this one's after the barrier.   */
static_assert(PGB_ITEMS * (PGB_PUSH_THREADS / 32) == 32, "a tile's list is 32 mask words");
__device__ __forceinline__ void tile_masks(const bool (&f)[PGB_ITEMS], int tile, unsigned* masks, int* tc,
                                           int* s_cnt, int& it) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int c = 0;
#pragma unroll
    for (int k = 0; k < PGB_ITEMS; ++k) {
        const unsigned m = __ballot_sync(0xffffffffu, f[k]);
        if (lane == 0) {
            masks[(long long)tile * 32 + k * (PGB_PUSH_THREADS / 32) + warp] = m;
            c += __popc(m);
        }
    }
    int* const cnt = &s_cnt[it & 1];
    if (lane == 0 && c) atomicAdd(cnt, c);
    __syncthreads();
    if (threadIdx.x == 0) {
        tc[tile] = *cnt;
        *cnt = 0;
    }
    ++it;
}

/* The shared deposit window holds each node's sum as one 32-bit word
 * (32-bit shared atomics are native, 64-bit ones are not).  A piece holds
 * at most PGB_PIECE_TILES * PGB_TILE = 4096 particles, and a contribution
 * of weight w < 1.99 is at most 1.99 * 2^19 + 1/2, so a node's sum stays
 * below 2^32.
 * Other weights deposit straight into the global int64 grid.  Both paths
 * add the same integer round(a*w*2^19).                                  */
#define WIN_NODES (PGB_WIN * PGB_WIN)
#define WIN_MAX_WEIGHT 1.99f
static_assert(PGB_PIECE_TILES * PGB_TILE <= 4096, "window sums are sized for 4096 particles per piece");
static_assert((PGB_FIX_SCALE * 1.99 + 1.0) * 4096.0 < 4294967296.0, "window sums must fit 32 bits");

/* deposit into the CTA's shared window when the four nodes fall inside it,
 * else into the global grid.  Caller checks deposit_ok (x, y > 0).       */
__device__ __forceinline__ void deposit_win(unsigned long long* qacc, unsigned int* win, int ox, int oy, int nx,
                                            int ps, float xs, float ys, float w) {
    const int jp = pbits(xs) >> ps, kp = pbits(ys) >> ps;
    const int lx = jp - ox, ly = kp - oy;
    /* 0 <= w < WIN_MAX_WEIGHT: such floats order as their bits, others' are above */
    if ((unsigned)lx < (unsigned)(PGB_WIN - 1) && (unsigned)ly < (unsigned)(PGB_WIN - 1) &&
        (unsigned)__float_as_int(w) < (unsigned)__float_as_int(WIN_MAX_WEIGHT)) {
        float wj = pfrac(xs, ps), wk = pfrac(ys, ps);
        float a4 = (1.0f - wj) * (1.0f - wk), a3 = wj * (1.0f - wk);
        float a2 = wk * (1.0f - wj), a1 = wj * wk;
        /* (a*w)*2^19 == a*(w*2^19) exactly: scaling by a power of two
         * commutes with rounding (w < 2: no overflow; a product below
         * FP32's normal range rounds to 0 either way)                     */
        const float wS = w * PGB_FIX_SCALE_F;
        const int k = ly * PGB_WIN + lx;
        /* below 2^21: the same integer as __float2ll_rn in deposit_cell */
        atomicAdd(&win[k], round_small(__fmul_rn(a4, wS)));
        atomicAdd(&win[k + 1], round_small(__fmul_rn(a3, wS)));
        atomicAdd(&win[k + PGB_WIN], round_small(__fmul_rn(a2, wS)));
        atomicAdd(&win[k + PGB_WIN + 1], round_small(__fmul_rn(a1, wS)));
    } else {
        deposit_cell(qacc, nx, ps, xs, ys, w);
    }
}

/* the same into a window of the whole grid, whose sums may wrap: pgb_deposit.cuh */
__device__ __forceinline__ void deposit_whole(unsigned long long* qacc, unsigned int* win, int nx, int ny, int ps,
                                              float xs, float ys, float w) {
    if ((unsigned)__float_as_int(w) >= (unsigned)__float_as_int(WIN_MAX_WEIGHT)) {
        deposit_cell(qacc, nx, ps, xs, ys, w);
        return;
    }
    const DepWindow W{win, 0, 0, nx, ny, true};
    const int k = (pbits(ys) >> ps) * nx + (pbits(xs) >> ps);
    const float wj = pfrac(xs, ps), wk = pfrac(ys, ps), wS = w * PGB_FIX_SCALE_F;
    dep_add(W, qacc, nx, k, (1.0f - wj) * (1.0f - wk), wS);
    dep_add(W, qacc, nx, k + 1, wj * (1.0f - wk), wS);
    dep_add(W, qacc, nx, k + nx, wk * (1.0f - wj), wS);
    dep_add(W, qacc, nx, k + nx + 1, wj * wk, wS);
}

/* ABSORB: a particle that leaves is removed here (and counted), where the
 * walls would do nothing else with it; else its tile's wall list is made */
template <bool DEP, bool ABSORB, bool WHOLE>
__device__ __forceinline__ void push_tile(const PushArgs& a, const PushConsts& pc, int tile, long long n,
                                          unsigned int* win, int ox, int oy, int* s_cnt, int& it, int& gone) {
    const long long base = (long long)tile * PGB_TILE;
    const int left = (int)min((long long)PGB_TILE, n - base);   /* slots of the tile in use */
    float4* const xv = a.xv + base;
    bool f[PGB_ITEMS];
    /* all loads of the thread's items first, so that they are in flight
     * together, then the pushes                                          */
    float4 p[PGB_ITEMS];
    float vz[PGB_ITEMS], w[PGB_ITEMS];
#pragma unroll
    for (int k = 0; k < PGB_ITEMS; ++k) {
        const int o = k * PGB_PUSH_THREADS + threadIdx.x;
        p[k] = make_float4(pos_dead(), 0.0f, 0.0f, 0.0f);
        vz[k] = 0.0f;
        w[k] = 0.0f;
        if (o < left) {
            p[k] = xv[o];
            if (pc.bfield) vz[k] = a.vz[base + o];
            if (DEP) w[k] = a.w[base + o];
        }
    }
#pragma unroll
    for (int k = 0; k < PGB_ITEMS; ++k) {
        f[k] = false;
        bool straight = false;   /* deposits straight to the grid */
        const int o = k * PGB_PUSH_THREADS + threadIdx.x;
        if (!is_dead(p[k].x)) {
            bool moved;
            gather_push_one(pc, a.exy, p[k], vz[k], moved);
            /* inside the deposit region it is outside no wall */
            if (deposit_ok(p[k].x, p[k].y, pc.nx, pc.ny, pc.ps)) {
                if (DEP && WHOLE) deposit_whole(a.qacc, win, pc.nx, pc.ny, pc.ps, p[k].x, p[k].y, w[k]);
                else if (DEP && win) deposit_win(a.qacc, win, ox, oy, pc.nx, pc.ps, p[k].x, p[k].y, w[k]);
                else straight = true;
            } else {
                f[k] = pc.steady ? outside_steady(p[k].x, p[k].y, pc.nx, pc.ny, pc.ps)
                                 : outside_absorbing(p[k].x, p[k].y, pc.nx, pc.ny, pc.ps);
                if (ABSORB && f[k]) {
                    p[k].x = pos_dead();
                    gone++;
                    moved = true;
                }
            }
            if (moved) xv[o] = p[k];
            if (pc.bfield && moved) a.vz[base + o] = vz[k];
        }
        if (DEP && !WHOLE && !win) deposit_pairs(a.qacc, pc.nx, pc.ps, straight, p[k].x, p[k].y, w[k]);
    }
    if (!ABSORB) tile_masks(f, tile, (unsigned*)a.tl_out, a.tc_out, s_cnt, it);
}

/* The window's non-zero sums to the grid, zeroed for the next piece.  A warp
 * per row; a lane takes columns lane and lane + 32, whose places in the
 * grid and whether they lie inside it are the same in every row.  (With
 * addresses and four bounds formed per node, the flush was 17% of the
 * push's instructions.)                                                  */
static_assert(PGB_WIN > 32 && PGB_WIN <= 64, "two columns a lane");
__device__ __forceinline__ void flush_window(unsigned long long* qacc, unsigned int* win, int ox, int oy, int nx, int ny) {
    const int lane = threadIdx.x & 31;
    const bool in0 = (unsigned)(ox + lane) < (unsigned)nx;
    const bool two = lane < PGB_WIN - 32, in1 = two && (unsigned)(ox + lane + 32) < (unsigned)nx;
    int ry = threadIdx.x >> 5;
    unsigned int* w = win + ry * PGB_WIN + lane;
    unsigned long long* q = qacc + (long long)(oy + ry) * nx + ox + lane;   /* used inside the grid only */
    const long long dq = (long long)(PGB_PUSH_THREADS / 32) * nx;
#pragma unroll
    for (int k = 0; k < (PGB_WIN + PGB_PUSH_THREADS / 32 - 1) / (PGB_PUSH_THREADS / 32); ++k) {
        if (ry < PGB_WIN) {
            const unsigned int v0 = w[0], v1 = two ? w[32] : 0u;
            const bool in = (unsigned)(oy + ry) < (unsigned)ny;
            if (v0) {
                w[0] = 0u;
                if (in && in0) atomicAdd(q, (unsigned long long)v0);
            }
            if (v1) {
                w[32] = 0u;
                if (in && in1) atomicAdd(q + 32, (unsigned long long)v1);
            }
        }
        ry += PGB_PUSH_THREADS / 32;
        w += PGB_PUSH_THREADS / 32 * PGB_WIN;
        q += dq;
    }
}

/* Work items: the bin pieces of the last sort (tiles of one bin, deposited
 * through a shared window), then every tile after the sorted region.
 * WHOLE: one window of the whole grid per block, flushed at its end.     */
template <bool DEP, bool ABSORB, bool WHOLE>
__global__ void __launch_bounds__(PGB_PUSH_THREADS, WHOLE ? 2 : 4) k_push(PushArgs a) {
    pgb_pdl_entry();
    __shared__ unsigned int s_win[WHOLE ? 1 : WIN_NODES];
    extern __shared__ __align__(16) unsigned int s_grid[];   /* WHOLE */
    const long long n = a.ds->n[a.s];
    const int ntiles = (int)((n + PGB_TILE - 1) / PGB_TILE);
    const int npieces = a.ds->n_pieces[a.s];
    const int tile0 = (int)a.ds->sorted_tiles[a.s];
    const int nitems = npieces + (ntiles > tile0 ? ntiles - tile0 : 0);
    if ((int)blockIdx.x >= nitems) return;   /* small runs: no item for this block */
    const PushConsts pc = a.pc;
    __shared__ int s_cnt[2];
    int it = 0, gone = 0;
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
    /* the window starts zeroed; each flush leaves it zeroed again */
    if (WHOLE)
        for (int k = threadIdx.x; k < pc.nx * pc.ny; k += blockDim.x) s_grid[k] = 0u;
    else if (DEP && npieces > 0)
        for (int k = threadIdx.x; k < WIN_NODES; k += blockDim.x) s_win[k] = 0u;
    __syncthreads();
    /* A block's first item is its own; where there are more items than
     * blocks, the others come from a counter: a fixed share of the pieces
     * left the SMs between 75 and 117% of their mean work (4 Mi electrons at
     * 513^2).  The next item is fetched while the present one is in work.
     * Without pieces the items are single tiles, alike, and shared out.    */
    const bool more = npieces > 0 && nitems > (int)gridDim.x;
    __shared__ int s_item[2];
    int turn = 0;
    for (int item = blockIdx.x; item < nitems; turn ^= 1) {
        if (more && threadIdx.x == 0) s_item[turn] = (int)gridDim.x + atomicAdd(&a.ds->work[a.s], 1);
        if (item < npieces) {
            int4 pc4 = a.pieces[item];
            unsigned int* win = nullptr;
            int ox = 0, oy = 0;
            if (WHOLE) {
                win = s_grid;
            } else if (DEP && pc4.z >= 0) {
                win = s_win;
                ox = (pc4.z % a.nbx) * PGB_BIN - PGB_HALO;
                oy = (pc4.z / a.nbx) * PGB_BIN - PGB_HALO;
            }
            for (int t = pc4.x; t < pc4.x + pc4.y && t < ntiles; ++t)
                push_tile<DEP, ABSORB, WHOLE>(a, pc, t, n, win, ox, oy, s_cnt, it, gone);
            if (!WHOLE && win) {
                __syncthreads();
                flush_window(a.qacc, s_win, ox, oy, pc.nx, pc.ny);
                __syncthreads();
            }
        } else {
            push_tile<DEP, ABSORB, WHOLE>(a, pc, tile0 + (item - npieces), n, WHOLE ? s_grid : nullptr, 0, 0, s_cnt, it, gone);
        }
        if (!more) {
            item += gridDim.x;
            continue;
        }
        __syncthreads();   /* the next item is there, and the other word is free */
        item = s_item[turn];
    }
    if (WHOLE) {
        __syncthreads();
        for (int row = threadIdx.x >> 5; row < pc.ny; row += PGB_PUSH_THREADS / 32)
            for (int c = threadIdx.x & 31; c < pc.nx; c += 32) {
                const unsigned int v = s_grid[row * pc.nx + c];
                if (v) atomicAdd(a.qacc + (long long)row * pc.nx + c, (unsigned long long)v);
            }
    }
    /* the last block to get here puts the counter back */
    if (more && threadIdx.x == 0 && atomicAdd(&a.ds->work_done[a.s], 1) == (int)gridDim.x - 1) {
        a.ds->work[a.s] = 0;
        a.ds->work_done[a.s] = 0;
    }
    if (ABSORB) {
        gone = __reduce_add_sync(0xffffffffu, gone);
        if ((threadIdx.x & 31) == 0 && gone) {
            atomicAdd((unsigned long long*)&a.ds->dead[a.s], (unsigned long long)gone);
            atomicAdd((unsigned long long*)&a.ds->stats[a.s == 0 ? ST_ABS_E : ST_ABS_I], (unsigned long long)gone);
        }
    }
}

/* flag-only pass (wall classification without a push) */
__global__ void __launch_bounds__(PGB_PUSH_THREADS) k_flag(const float4* xv, DevState* ds, int s, int nx, int ny,
                                                           int ps, int steady, int* tl, int* tc) {
    pgb_pdl_entry();
    const long long n = ds->n[s];
    const int ntiles = (int)((n + PGB_TILE - 1) / PGB_TILE);
    __shared__ int s_cnt[2];
    int it = 0;
    if (threadIdx.x < 2) s_cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long base = (long long)tile * PGB_TILE;
        bool f[PGB_ITEMS];
#pragma unroll
        for (int k = 0; k < PGB_ITEMS; ++k) {
            long long i = base + k * PGB_PUSH_THREADS + threadIdx.x;
            f[k] = false;
            if (i >= n) continue;
            float4 p = xv[i];
            if (is_dead(p.x)) continue;
            f[k] = steady ? outside_steady(p.x, p.y, nx, ny, ps) : outside_absorbing(p.x, p.y, nx, ny, ps);
        }
        tile_masks(f, tile, (unsigned*)tl, tc, s_cnt, it);
    }
}

/* standalone deposit (particle::collect_charge) */
struct SlotSource {
    const float4* xv;
    const float* w;
    __device__ __forceinline__ void operator()(long long i, float& x, float& y, float& wt) const {
        const float4 p = xv[i];
        x = p.x;
        y = p.y;
        wt = w[i];
    }
};
/* few particles for the grid: a thread each, straight to the accumulator */
__global__ void __launch_bounds__(256) k_deposit_few(SlotSource src, const DevState* ds, int s, int nx, int ny, int ps,
                                                     unsigned long long* qacc) {
    pgb_pdl_entry();
    const long long n = ds->n[s];
    for (long long base = blockIdx.x * 256ll; base < n; base += gridDim.x * 256ll) {
        const long long i = base + threadIdx.x;
        float x = pos_dead(), y = pos_dead(), w = 0.0f;
        if (i < n) src(i, x, y, w);
        deposit_pairs(qacc, nx, ps, deposit_ok(x, y, nx, ny, ps), x, y, w);
    }
}
__global__ void __launch_bounds__(DEP_THREADS) k_deposit(SlotSource src, DevState* ds, int s, int nx, int ny, int ps,
                                                         unsigned long long* qacc) {
    pgb_pdl_entry();
    deposit_windows(src, ds->n[s], nx, ny, ps, qacc);
}

/* e_collisions::collision (e_collisions.cpp:480-597), the first kernel of a
 * step: the collision test of every electron, the scatterings (about one
 * electron in twenty), the ionizations' effect on their parents, and the
 * ionization events' number or their ordered per-tile list.  It reads no
 * field, so it runs while the previous step's field solve is in flight.
 * Each event touches only its own electron and draws from that electron's
 * stream, so the order in which events are handled changes nothing.
 *
 * Every warp works alone, on 128 consecutive slots at a time:
 *   (1) every electron: the domain test, |v|^2, the Philox draw R and
 *       mcc_candidate; the candidates (about one in ten at a few eV) go to
 *       the warp's queue in shared memory;
 *   (2) whenever 32 candidates wait, one per lane: the cross-sections, the
 *       exponential and the decisions of mcc_decide; the scatterings go to
 *       a second queue;
 *   (3) whenever 32 scatterings wait, one per lane: the electron (read
 *       again, from L1 or L2) scatters and, if it also ionizes, ionizes.
 * Bound by instruction issue: one Philox4x32-10 block per electron is
 * about half of it.  With a tile per 256 threads, queues per tile, five
 * barriers a tile and the scatterings in a kernel of their own it took 145
 * + 28 us at 16 Mi electrons.
 *
 * At 64 registers a thread a block fills an SM's register file, so a grid
 * of sms - k blocks leaves k SMs wholly free for the field solve beside it. */
#define MCC_GROUPS 4                                    /* tiles a block has in work  */
#define MCC_THREADS (MCC_GROUPS * PGB_PUSH_THREADS)
#define MCC_WARPS (MCC_THREADS / 32)
#define MCC_UNIT 128                                    /* slots of a warp at a time  */
#define MCC_ION_BIT 0x80000000u
static_assert(MCC_UNIT * (PGB_PUSH_THREADS / 32) == PGB_TILE, "eight warps share a tile");
struct MccQueue {
    float u2[32 + MCC_UNIT], r[32 + MCC_UNIT];   /* candidates: |v|^2, R, slot */
    int slot[32 + MCC_UNIT];
    unsigned scat[64];                           /* scatterings: slot | MCC_ION_BIT */
};
/* one candidate per lane of the first m: decisions; returns the number of
 * scatterings queued                                                     */
__device__ __forceinline__ int mcc_candidates(const PushArgs& a, MccQueue& Q, int base, int m, int nscat, unsigned step,
                                              int (&st)[2], bool list) {
    const int lane = threadIdx.x & 31;
    int ev = 0, slot = 0;
    if (lane < m) {
        slot = Q.slot[base + lane];
        ev = mcc_decide(a.cc, Q.u2[base + lane], Q.r[base + lane]);
    }
    const bool sc = (ev & MCC_SCATTER) != 0, io = (ev & MCC_IONIZE) != 0;
    st[0] += sc ? 1 : 0;
    st[1] += io ? 1 : 0;
    if (io) {
        if (list) {
            /* slot order: word slot/32 of the lists, bit slot%32 (tile_masks) */
            atomicOr((unsigned*)a.tl_ev + (slot >> 5), 1u << (slot & 31));
            atomicAdd(a.tc_ev + slot / PGB_TILE, 1);
        }
        if (!sc) {
            float4 p = a.xv[slot];
            float vz = a.vz[slot];
            mcc_ionize(a.cc, a.neut, a.id[slot], step, p, vz);
            a.xv[slot] = p;
            a.vz[slot] = vz;
        }
    }
    const unsigned ms = __ballot_sync(0xffffffffu, sc);
    if (sc) Q.scat[nscat + __popc(ms & ((1u << lane) - 1u))] = (unsigned)slot | (io ? MCC_ION_BIT : 0u);
    __syncwarp();
    return nscat + __popc(ms);
}
/* one scattering per lane of the first m */
__device__ __forceinline__ void mcc_scatterings(const PushArgs& a, const MccQueue& Q, int base, int m, unsigned step) {
    const int lane = threadIdx.x & 31;
    if (lane < m) {
        const unsigned e = Q.scat[base + lane];
        const int slot = (int)(e & ~MCC_ION_BIT);
        float4 p = a.xv[slot];
        float vz = a.vz[slot];
        const unsigned int id = a.id[slot];
        const float energy = a.cc.e_energy_coef * speed2(p, vz);
        pgb_stream st;
        pgb_stream_init(&st, a.cc.seed, id, step, PGB_STREAM_EMCC, 0);
        (void)pgb_stream_u32(&st);   /* the collision test's draw */
        scatter_f32(&st, a.neut, a.cc.n_neutral, energy, (float)a.cc.reduced_mass, p.z, p.w, vz);
        if (e & MCC_ION_BIT) mcc_ionize(a.cc, a.neut, id, step, p, vz);
        a.xv[slot] = p;
        a.vz[slot] = vz;
    }
    __syncwarp();
}
__global__ void __launch_bounds__(MCC_THREADS, 1) k_mcc(PushArgs a, int list) {
    pgb_pdl_entry();
    extern __shared__ __align__(16) unsigned char s_mcc[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    MccQueue& Q = reinterpret_cast<MccQueue*>(s_mcc)[warp];
    const long long n = a.ds->n[0];
    const int ntiles = (int)((n + PGB_TILE - 1) / PGB_TILE);
    const unsigned step = (unsigned)a.ds->t;
    int st_loc[2] = {0, 0};
    int nc = 0, ns = 0;   /* candidates and scatterings queued */
    for (int tile = blockIdx.x * MCC_GROUPS + (warp >> 3); tile < ntiles; tile += gridDim.x * MCC_GROUPS) {
        const int base = tile * PGB_TILE + (warp & 7) * MCC_UNIT;
        const int left = (int)min((long long)MCC_UNIT, n - base);   /* slots of this unit in use */
        if (left <= 0 && !list) continue;
        /* all loads of the lane's items first, then the draws */
        float4 pa[MCC_UNIT / 32];
        float vza[MCC_UNIT / 32];
        unsigned int ida[MCC_UNIT / 32];
#pragma unroll
        for (int k = 0; k < MCC_UNIT / 32; ++k) {
            const int o = k * 32 + lane;
            pa[k] = make_float4(pos_dead(), 0.0f, 0.0f, 0.0f);
            vza[k] = 0.0f;
            ida[k] = 0u;
            if (o < left) {
                pa[k] = a.xv[base + o];
                vza[k] = a.vz[base + o];
                ida[k] = a.id[base + o];
            }
        }
        if (list && lane < MCC_UNIT / 32) ((unsigned*)a.tl_ev)[(base >> 5) + lane] = 0u;
#pragma unroll
        for (int k = 0; k < MCC_UNIT / 32; ++k) {
            float u2 = 0.0f, R = 1.0f;
            bool c = false;
            if (!is_dead(pa[k].x) && mcc_draw(a.cc, ida[k], step, a.pc.nx, a.pc.ny, a.pc.ps, pa[k], vza[k], u2, R))
                c = mcc_candidate(a.cc, u2, R);
            const unsigned cm = __ballot_sync(0xffffffffu, c);
            if (c) {
                const int q = nc + __popc(cm & lt);
                Q.u2[q] = u2;
                Q.r[q] = R;
                Q.slot[q] = base + k * 32 + lane;
            }
            nc += __popc(cm);
        }
        __syncwarp();
        /* the queues from their ends, so that what stays is in place */
        while (nc >= 32) {
            nc -= 32;
            ns = mcc_candidates(a, Q, nc, 32, ns, step, st_loc, list);
            if (ns >= 32) {
                ns -= 32;
                mcc_scatterings(a, Q, ns, 32, step);
            }
        }
    }
    if (nc) ns = mcc_candidates(a, Q, 0, nc, ns, step, st_loc, list);
    for (int q = 0; q < ns; q += 32) mcc_scatterings(a, Q, q, min(32, ns - q), step);
    flush_stats(st_loc, a.ds->stats, list ? nullptr : &a.ds->list_n[LIST_ION_EV]);
}

/* the last kernel of a step's particle phases moves the step counter on
 * (where the wall kernels do not, see pgb_launch_walls); commit: species
 * whose uncounted ionization products it enters                          */
__global__ void k_step_advance(DevState* ds, int commit) {
    pgb_pdl_entry();
    if (commit) ionize_count_commit(ds, commit);
    pgb_step_end(ds);
}

/* ------------------------------------------------------------ scans */
/* exclusive scan of cnt[0..m) into off[]; returns the total.  One block of
 * 1024 threads, 8 consecutive items per thread and 8192 entries per pass.
 * (32 items per thread, one pass for the bench's 16.7K tiles, measured
 * slower: a warp's load then touches 32 lines instead of 8.)            */
#define SCAN_ITEMS 8
__device__ __forceinline__ long long block_excl_scan(const int* cnt, int* off, long long m, long long carry0) {
    __shared__ long long s_warp[32];
    __shared__ long long s_carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_carry = carry0;
    __syncthreads();
    for (long long b = 0; b < m; b += SCAN_ITEMS * 1024) {
        long long i0 = b + SCAN_ITEMS * (long long)threadIdx.x;
        int v[SCAN_ITEMS];
        long long sum = 0;
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS; ++q) v[q] = (i0 + q < m) ? cnt[i0 + q] : 0;
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS; ++q) sum += v[q];
        long long x = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            long long y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) s_warp[warp] = x;
        __syncthreads();
        if (warp == 0) {
            long long t = s_warp[lane];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                long long y = __shfl_up_sync(0xffffffffu, t, d);
                if (lane >= d) t += y;
            }
            s_warp[lane] = t;
        }
        __syncthreads();
        long long excl = s_carry + (warp ? s_warp[warp - 1] : 0) + x - sum;
#pragma unroll
        for (int q = 0; q < SCAN_ITEMS; ++q) {
            if (i0 + q < m) off[i0 + q] = (int)excl;
            excl += v[q];
        }
        __syncthreads();
        if (threadIdx.x == 0) s_carry += s_warp[31];
        __syncthreads();
    }
    return s_carry;
}

__global__ void __launch_bounds__(1024) k_scan_small(const int* cnt, int* off, const long long* n_ptr, long long m_const,
                                                     long long* total) {
    pgb_pdl_entry();
    /* n_ptr: particle count whose tiles are scanned; else m_const entries */
    const long long m = n_ptr ? (*n_ptr + PGB_TILE - 1) / PGB_TILE : m_const;
    long long t = block_excl_scan(cnt, off, m, 0);
    if (threadIdx.x == 0) *total = t;
}

/* Per-tile lists (32 mask words a tile, see tile_masks) to one dense list
 * in slot order, and its length, in one launch.  A block takes a run of
 * tiles; the entries before its first tile are the sum of the counts
 * before it, which every block adds up for itself (at 16.4 Ki tiles 32 KB
 * from L2 on average), so that no block waits for another.  A warp per
 * tile, a lane per word: a shuffle scan of the words' counts gives each
 * word's place, then each lane writes the slots of its set bits.
 * One launch instead of a one-block scan and a gather: at 16.4 Ki tiles
 * 15.7 + 5.9 us -> 7 us, at 200 tiles 4.1 + 3.6 -> 4 us (ncu).
 * commit: species whose uncounted ionization products this list's last
 * block enters (0: none).                                                */
#define LIST_THREADS 512
__global__ void __launch_bounds__(LIST_THREADS) k_build_list(const int* tl, const int* tc, DevState* ds, int s, int* out,
                                                             long long* total, int commit) {
    pgb_pdl_entry();
    __shared__ int s_sum[LIST_THREADS / 32];
    __shared__ int s_off[LIST_THREADS];
    const int ntiles = (int)((ds->n[s] + PGB_TILE - 1) / PGB_TILE);
    const int per = (ntiles + gridDim.x - 1) / gridDim.x;
    const int t0 = min((int)blockIdx.x * per, ntiles), t1 = min(t0 + per, ntiles);
    const bool last = t1 == ntiles && (t0 < t1 || blockIdx.x == 0);
    if (t0 == t1 && !last) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned* masks = (const unsigned*)tl;
    int sum = 0;
    for (int t = threadIdx.x; t < t0; t += LIST_THREADS) sum += tc[t];
#pragma unroll
    for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0) s_sum[warp] = sum;
    __syncthreads();
    int carry = 0;
#pragma unroll
    for (int w = 0; w < LIST_THREADS / 32; ++w) carry += s_sum[w];
    for (int b = t0; b < t1; b += LIST_THREADS) {
        /* exclusive scan of this run's counts */
        const int c = b + (int)threadIdx.x < t1 ? tc[b + threadIdx.x] : 0;
        int x = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        __syncthreads();   /* s_sum and s_off of the pass before have been read */
        if (lane == 31) s_sum[warp] = x;
        __syncthreads();
        int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < LIST_THREADS / 32; ++w) {
            if (w < warp) before += s_sum[w];
            all += s_sum[w];
        }
        s_off[threadIdx.x] = carry + before + x - c;
        __syncthreads();
        const int m1 = min(b + LIST_THREADS, t1);
        for (int t = b + warp; t < m1; t += LIST_THREADS / 32) {
            unsigned m = masks[(long long)t * 32 + lane];
            const int cw = __popc(m);
            int incl = cw;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += y;
            }
            int pos = s_off[t - b] + incl - cw;
            /* word lane = k * warps + w holds slots tile*TILE + k*THREADS + w*32 + bit */
            const int sb = t * PGB_TILE + (lane / (PGB_PUSH_THREADS / 32)) * PGB_PUSH_THREADS +
                           (lane % (PGB_PUSH_THREADS / 32)) * 32;
            while (m) {
                const int q = __ffs(m) - 1;
                m &= m - 1;
                out[pos++] = sb + q;
            }
        }
        carry += all;
    }
    if (last && threadIdx.x == 0) {
        *total = carry;
        if (commit) ionize_count_commit(ds, commit);
    }
}

/* ------------------------------------------------------------ inject */
/* particle::inject_more_particles (particle.cpp:491-510): uniform position
 * in [DX, L-DX]^2, velocities from get_particle_velocity, weight 0.0.  For
 * electrons the new particles are pushed here too (they are created before
 * the electron push in pic_run, after the collision loop).               */
struct InjectArgs {
    Species e, i;
    DevState* ds;
    int k;                       /* NUMBER_TO_INJECT */
    double dx, dy, xlength, ylength;
    uint64_t seed;
    PushConsts pce;
    const float2* exy;
    int push_e;                  /* push the new electrons (inside pgb_step) */
    int absorb_e;                /* ... and remove those that leave          */
    int species_mask;            /* 1 = electrons, 2 = ions                  */
    int* list_out_e;             /* append outside electrons (ordered)       */
    long long list_cap;
    int* flag;                   /* k_inject: per new electron, outside after its push */
};
/* the j-th new particle of species s: id and slot from the counts before
 * the injection; true if it left through a wall in its first push        */
__device__ __forceinline__ bool inject_one(const InjectArgs& a, int s, int jj, long long n0, unsigned int id0) {
    const Species& S = s == 0 ? a.e : a.i;
    const long long slot = n0 + jj;
    if (slot >= S.cap) { atomicOr(&a.ds->err, s == 0 ? ERR_CAP_E : ERR_CAP_I); return false; }
    const unsigned int id = id0 + (unsigned int)jj;
    pgb_stream st;
    pgb_stream_init(&st, a.seed, id, (unsigned int)a.ds->t, PGB_STREAM_INJECT, (uint32_t)s);
    double rx = pgb_u01d(pgb_stream_u32(&st));
    double ry = pgb_u01d(pgb_stream_u32(&st));
    double x = (a.dx + rx * (a.xlength - 2.0 * a.dx));
    double y = (a.dy + ry * (a.ylength - 2.0 * a.dy));
    float vt = (float)S.vt;
    float vx = maxwell_f32(&st, vt), vy = maxwell_f32(&st, vt), vz = maxwell_f32(&st, vt);
    float4 p = make_float4(pos_from_m(x, a.dx, a.pce.ps), pos_from_m(y, a.dy, a.pce.ps), vx, vy);
    bool out = false;
    if (s == 0 && a.push_e) {
        bool moved;
        gather_push_one(a.pce, a.exy, p, vz, moved);
        /* weight 0: the deposit adds nothing (particle.cpp:497) */
        out = a.pce.steady ? outside_steady(p.x, p.y, a.pce.nx, a.pce.ny, a.pce.ps)
                           : outside_absorbing(p.x, p.y, a.pce.nx, a.pce.ny, a.pce.ps);
        if (out && a.absorb_e) {
            p.x = pos_dead();
            atomicAdd((unsigned long long*)&a.ds->dead[0], 1ull);
            atomicAdd((unsigned long long*)&a.ds->stats[ST_ABS_E], 1ull);
            out = false;   /* joins no list */
        }
    }
    S.xv[slot] = p;
    S.vz[slot] = vz;
    S.w[slot] = 0.0f;
    S.id[slot] = id;
    return out;
}
__global__ void k_inject(InjectArgs a) {
    pgb_pdl_entry();
    /* one thread per new particle; electrons first, then ions, in id order */
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int total = a.k * ((a.species_mask & 1) + ((a.species_mask >> 1) & 1));
    if (j >= total) return;
    const int s = ((a.species_mask & 1) && j < a.k) ? 0 : 1;
    const int jj = (s == 0 || !(a.species_mask & 1)) ? j : j - a.k;
    /* outside electrons join the end of the wall list in slot order */
    if (inject_one(a, s, jj, a.ds->n[s], a.ds->next_id[s])) a.flag[jj] = 1;
}

/* The injection of one species in one block, for NUMBER_TO_INJECT up to
 * INJECT_BLOCK_MAX: the ids of the step's uncounted ionization products
 * first (commit), the particles, then the counts and the wall list.  Two
 * launches and the products' commit kernel in one (6.4 + 4.2 + 2.3 us ->
 * 6.5 us, ncu).  More particles are better spread over blocks (k_inject):
 * each one's draws and divisions keep an SM's FP64 pipe busy.  A step with
 * one block / spread: 10 injected 70.5 / 72.0 us, 200 74.9 / 73.9, 600 84.6
 * / 75.6, 1000 102 / 79, 4000 183 / 83.                                   */
#define INJECT_BLOCK_MAX 256
__global__ void __launch_bounds__(INJECT_BLOCK_MAX) k_inject_block(InjectArgs a, int s, int commit) {
    pgb_pdl_entry();
    __shared__ unsigned s_out[INJECT_BLOCK_MAX / 32];
    if (commit && threadIdx.x == 0) ionize_count_commit(a.ds, commit);
    __syncthreads();
    const Species& S = s == 0 ? a.e : a.i;
    const long long n0 = a.ds->n[s];
    const unsigned int id0 = a.ds->next_id[s];
    for (int j = threadIdx.x; j < ((a.k + 31) & ~31); j += blockDim.x) {
        const bool out = j < a.k && inject_one(a, s, j, n0, id0);
        const unsigned m = __ballot_sync(0xffffffffu, out);
        if ((threadIdx.x & 31) == 0) s_out[j >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    int k = a.k;
    if (n0 + k > S.cap) k = (int)(S.cap - n0 > 0 ? S.cap - n0 : 0);
    if (s == 0 && a.push_e) {
        long long pos = a.ds->list_n[LIST_OUT_E];
        for (int w = 0; w < (k + 31) / 32; ++w)
            for (unsigned m = s_out[w]; m; m &= m - 1) {
                const int j = 32 * w + __ffs(m) - 1;
                if (pos < a.list_cap) a.list_out_e[pos++] = (int)(n0 + j);
                else atomicOr(&a.ds->err, ERR_LIST);   /* the ions' injection may report beside it */
            }
        a.ds->list_n[LIST_OUT_E] = pos;
    }
    a.ds->n[s] = n0 + k;
    a.ds->next_id[s] = id0 + (unsigned int)k;
    a.ds->stats[s == 0 ? ST_INJ_E : ST_INJ_I] += k;
}

/* after k_inject: counts, ids, and the wall list entries of new electrons in
 * slot order, 1024 flags at a time (one thread took 261 us for 5000)      */
__global__ void __launch_bounds__(1024) k_inject_commit(InjectArgs a) {
    pgb_pdl_entry();
    __shared__ int s_cnt[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int s = 0; s < 2; ++s) {
        if (!(a.species_mask & (1 << s))) continue;
        const Species& S = s == 0 ? a.e : a.i;
        const long long n0 = a.ds->n[s];
        int k = a.k;
        if (n0 + k > S.cap) k = (int)(S.cap - n0 > 0 ? S.cap - n0 : 0);
        if (s == 0 && a.push_e && !a.absorb_e) {
            long long pos = a.ds->list_n[LIST_OUT_E];
            for (int base = 0; base < k; base += 1024) {
                const int j = base + threadIdx.x;
                const bool f = j < k && a.flag[j];
                const unsigned m = __ballot_sync(0xffffffffu, f);
                if (lane == 0) s_cnt[warp] = __popc(m);
                __syncthreads();
                int before = __popc(m & ((1u << lane) - 1u)), all = 0;
                for (int w = 0; w < 32; ++w) {
                    if (w < warp) before += s_cnt[w];
                    all += s_cnt[w];
                }
                if (f) {
                    a.flag[j] = 0;
                    if (pos + before < a.list_cap) a.list_out_e[pos + before] = (int)(n0 + j);
                    else atomicOr(&a.ds->err, ERR_LIST);
                }
                pos += all;
                __syncthreads();
            }
            if (threadIdx.x == 0) a.ds->list_n[LIST_OUT_E] = pos < a.list_cap ? pos : a.list_cap;
        }
        __syncthreads();   /* every thread has read the counts */
        if (threadIdx.x == 0) {
            a.ds->n[s] = n0 + k;
            a.ds->next_id[s] += (unsigned int)k;
            a.ds->stats[s == 0 ? ST_INJ_E : ST_INJ_I] += k;
        }
    }
}

/* ------------------------------------------------- ionization products */
/* e_collisions::ionization appends one ion and one electron per event
 * (e_collisions.cpp:406-441); both are NaN (see ionize_fp64).  With
 * absorbing walls the electron is removed by the wall pass of the same
 * step, and so is the ion on an ion step, so those are counted without
 * being stored; otherwise they are stored in event order.                 */
struct IonizeAppendArgs {
    Species e, i;
    DevState* ds;
    const int* ev;               /* dense event list (electron slots)      */
    CollConsts cc;
    const float* neut;
    double dx, dy;
    int ps;
    int store_e, store_i;
};
__global__ void k_ionize_append(IonizeAppendArgs a) {
    pgb_pdl_entry();
    const long long m = a.ds->list_n[LIST_ION_EV];
    const long long ne0 = a.ds->n[0], ni0 = a.ds->n[1];
    const unsigned int ide0 = a.ds->next_id[0], idi0 = a.ds->next_id[1];
    for (long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x; r < m; r += (long long)gridDim.x * blockDim.x) {
        if (!a.store_e && !a.store_i) break;
        int slot = a.ev[r];
        unsigned int pid = a.e.id[slot];
        /* recompute the event's products from the parent's stream; the
         * parent's pre-event velocity is not needed because every product
         * is NaN (the excess energy is negative)                           */
        pgb_stream si;
        pgb_stream_init(&si, a.cc.seed, pid, (unsigned int)a.ds->t, PGB_STREAM_IONIZE, 0);
        float4 pp = a.e.xv[slot];
        double xe = pos_m(pp.x, a.ps, a.dx), ye = pos_m(pp.y, a.ps, a.dy);
        IonizeOut o = ionize_f32(&si, a.neut, a.cc.n_neutral, a.cc, xe, ye, 0.0f, 0.0f, 0.0f);
        if (a.store_i) {
            long long s2 = ni0 + r;
            if (s2 < a.i.cap) {
                a.i.xv[s2] = make_float4(pos_from_m(o.ix, a.dx, a.ps), pos_from_m(o.iy, a.dy, a.ps), (float)o.ivx,
                                         (float)o.ivy);
                a.i.vz[s2] = (float)o.ivz;
                a.i.w[s2] = a.e.w[slot];
                a.i.id[s2] = idi0 + (unsigned int)r;
            } else {
                atomicOr(&a.ds->err, ERR_CAP_I);
            }
        }
        if (a.store_e) {
            long long s2 = ne0 + r;
            if (s2 < a.e.cap) {
                a.e.xv[s2] = make_float4(pos_from_m(o.nx_, a.dx, a.ps), pos_from_m(o.ny_, a.dy, a.ps), (float)o.nvx,
                                         (float)o.nvy);
                a.e.vz[s2] = (float)o.nvz;
                a.e.w[s2] = a.e.w[slot];
                a.e.id[s2] = ide0 + (unsigned int)r;
            } else {
                atomicOr(&a.ds->err, ERR_CAP_E);
            }
        }
    }
}
__global__ void k_ionize_commit(DevState* ds, int store_e, int store_i, long long cap_e, long long cap_i) {
    pgb_pdl_entry();
    long long m = ds->list_n[LIST_ION_EV];
    ds->next_id[0] += (unsigned int)m;
    ds->next_id[1] += (unsigned int)m;
    if (store_e) { long long v = ds->n[0] + m; ds->n[0] = v < cap_e ? v : cap_e; }
    else ds->stats[ST_ABS_E] += m;
    if (store_i) { long long v = ds->n[1] + m; ds->n[1] = v < cap_i ? v : cap_i; }
    else ds->stats[ST_ABS_I] += m;
    ds->list_n[LIST_ION_EV] = 0;   /* k_mcc counts on from 0 where no list is built */
}

__global__ void k_ionize_count_commit(DevState* ds, int species_mask) {
    pgb_pdl_entry();
    ionize_count_commit(ds, species_mask);
}

/* ------------------------------------------------------------ compaction */
__global__ void __launch_bounds__(PGB_PUSH_THREADS) k_alive_count(const float4* xv, DevState* ds, int s, int* tc) {
    pgb_pdl_entry();
    const long long n = ds->n[s];
    const int ntiles = (int)((n + PGB_TILE - 1) / PGB_TILE);
    __shared__ int s_w[PGB_PUSH_THREADS / 32];
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int c = 0;
        for (int k = 0; k < PGB_ITEMS; ++k) {
            long long i = (long long)tile * PGB_TILE + k * PGB_PUSH_THREADS + threadIdx.x;
            if (i < n && !is_dead(xv[i].x)) c++;
        }
        for (int d = 16; d; d >>= 1) c += __shfl_down_sync(0xffffffffu, c, d);
        if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            int t = 0;
            for (int w = 0; w < PGB_PUSH_THREADS / 32; ++w) t += s_w[w];
            tc[tile] = t;
        }
        __syncthreads();
    }
}
__global__ void __launch_bounds__(PGB_PUSH_THREADS) k_compact(Species S, DevState* ds, int s, const int* toff) {
    pgb_pdl_entry();
    const long long n = ds->n[s];
    const int ntiles = (int)((n + PGB_TILE - 1) / PGB_TILE);
    bool f[1][PGB_ITEMS];
    __shared__ int s_off[PGB_ITEMS][PGB_PUSH_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        unsigned m[PGB_ITEMS];
        for (int k = 0; k < PGB_ITEMS; ++k) {
            long long i = (long long)tile * PGB_TILE + k * PGB_PUSH_THREADS + threadIdx.x;
            f[0][k] = (i < n) && !is_dead(S.xv[i].x);
            m[k] = __ballot_sync(0xffffffffu, f[0][k]);
            if (lane == 0) s_off[k][warp] = __popc(m[k]);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int acc = toff[tile];
            for (int k = 0; k < PGB_ITEMS; ++k)
                for (int w = 0; w < PGB_PUSH_THREADS / 32; ++w) { int c = s_off[k][w]; s_off[k][w] = acc; acc += c; }
        }
        __syncthreads();
        for (int k = 0; k < PGB_ITEMS; ++k)
            if (f[0][k]) {
                long long i = (long long)tile * PGB_TILE + k * PGB_PUSH_THREADS + threadIdx.x;
                int pos = s_off[k][warp] + __popc(m[k] & ((1u << lane) - 1u));
                S.xv2[pos] = S.xv[i];
                S.vz2[pos] = S.vz[i];
                S.w2[pos] = S.w[i];
                S.id2[pos] = S.id[i];
            }
        __syncthreads();
    }
}
__global__ void k_compact_commit(DevState* ds, int s, const long long* total) {
    pgb_pdl_entry();
    ds->n[s] = *total;
    ds->dead[s] = 0;
    ds->n_pieces[s] = 0;       /* slot order changed: the bin pieces are gone */
    ds->sorted_tiles[s] = 0;
}

/* ------------------------------------------------------------ load / dump */
/* slots [i0, i1) from records aos[6 i ..] */
__global__ void k_load(Species S, const double* aos, long long i0, long long i1, double dx, double dy, PosScale rx, PosScale ry,
                       int ps) {
    pgb_pdl_entry();
    for (long long i = i0 + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < i1; i += (long long)gridDim.x * blockDim.x) {
        const double* r = aos + 6 * i;
        S.xv[i] = make_float4(pos_from_m(r[0], dx, rx, ps), pos_from_m(r[1], dy, ry, ps), (float)r[2], (float)r[3]);
        S.vz[i] = (float)r[4];
        S.w[i] = weight_from_double(r[5]);
        S.id[i] = (unsigned int)i;
    }
}
/* dump live slots in order: out[j] for the j-th live slot; pos[] = exclusive
 * scan of the per-tile live counts                                        */
/* tiles [t0, t1) of the live-slot order */
/* out (6 doubles per particle) and ids (the particle's id) are each
 * written when not null                                                  */
__global__ void __launch_bounds__(PGB_PUSH_THREADS) k_dump(Species S, DevState* ds, int s, const int* toff, double ux,
                                                           double uy, double* out, unsigned int* ids, long long cap,
                                                           int t0, int t1) {
    pgb_pdl_entry();
    const long long n = ds->n[s];
    const int ntiles = min(t1, (int)((n + PGB_TILE - 1) / PGB_TILE));
    __shared__ int s_off[PGB_ITEMS * (PGB_PUSH_THREADS / 32)];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int tile = t0 + blockIdx.x; tile < ntiles; tile += gridDim.x) {
        float4 p[PGB_ITEMS];
        bool f[PGB_ITEMS];
        unsigned m[PGB_ITEMS];
#pragma unroll
        for (int k = 0; k < PGB_ITEMS; ++k) {
            long long i = (long long)tile * PGB_TILE + k * PGB_PUSH_THREADS + threadIdx.x;
            p[k] = i < n ? S.xv[i] : make_float4(pos_dead(), 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int k = 0; k < PGB_ITEMS; ++k) {
            f[k] = !is_dead(p[k].x);
            m[k] = __ballot_sync(0xffffffffu, f[k]);
            if (lane == 0) s_off[k * (PGB_PUSH_THREADS / 32) + warp] = __popc(m[k]);
        }
        __syncthreads();
        if (warp == 0) {   /* 32 (item, warp) counts, a lane each */
            const int c = s_off[lane];
            int x = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            s_off[lane] = toff[tile] + x - c;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PGB_ITEMS; ++k)
            if (f[k]) {
                long long i = (long long)tile * PGB_TILE + k * PGB_PUSH_THREADS + threadIdx.x;
                long long pos = s_off[k * (PGB_PUSH_THREADS / 32) + warp] + __popc(m[k] & ((1u << lane) - 1u));
                if (pos < cap && out) {
                    double2* const o = reinterpret_cast<double2*>(out + 6 * pos);   /* 48 B a record, 16-byte aligned */
                    o[0] = make_double2(pos_m(p[k].x, ux), pos_m(p[k].y, uy));
                    o[1] = make_double2(f32_to_f64(p[k].z), f32_to_f64(p[k].w));
                    o[2] = make_double2(f32_to_f64(S.vz[i]), f32_to_f64(S.w[i]));
                }
                if (pos < cap && ids) ids[pos] = S.id[i];
            }
        __syncthreads();
    }
}

/* after a load: the species' counts; its slots are in no bin order */
__global__ void k_load_commit(DevState* ds, int s, long long n) {
    pgb_pdl_entry();
    ds->n[s] = n;
    ds->dead[s] = 0;
    ds->next_id[s] = (unsigned int)n;
    ds->n_pieces[s] = 0;
    ds->sorted_tiles[s] = 0;
}
/* the step counters, the right-wall potential of the first step where there
 * is only one (else the table is copied), and the ionization events counted
 * from 0 (a step that ended in an error leaves its count)                */
__global__ void k_set_step(DevState* ds, long long t, double* phi_tab, double phi, int one) {
    pgb_pdl_entry();
    ds->t = ds->t_base = ds->tf = t;
    if (one) phi_tab[0] = phi;
    ds->list_n[LIST_ION_EV] = 0;
}

/* ====================================================== host launchers */
static int grid_for(pgb_run* r, int per_sm) { return r->sms * per_sm; }

static PushConsts push_consts(pgb_run* r, int s) {
    PushConsts pc;
    const Species& S = r->sp[s];
    pc.nx = r->nx; pc.ny = r->ny;
    pc.ps = r->ps;
    pc.dtdx = (float)ldexp(S.dt / r->dx, r->ps);
    pc.dtdy = (float)ldexp(S.dt / r->dy, r->ps);
    pc.coef = (float)(0.5 * S.dt * S.q_over_m);
    double omega_dt = S.dt * S.q_over_m * r->p.magnetic_field;
    pc.ca = (float)cos(r->p.angle); pc.sa = (float)sin(r->p.angle);
    pc.co = (float)cos(omega_dt); pc.so = (float)sin(omega_dt);
    pc.bfield = r->p.magnetic_field > 0.0;
    pc.steady = r->p.steadystate;
    return pc;
}

/* the FP32 fits at the given energies (pgb_cross_sections) */
__global__ void k_cross_sections(int which, const double* e, long long n, double* out) {
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        const float x = (float)e[k];
        float s = 0.0f;
        switch (which) {
            case PGB_XS_AR_ELASTIC: s = sig_ar_el(x); break;
            case PGB_XS_AR_IONIZE: s = sig_ar_ion(x); break;
            case PGB_XS_H_ELASTIC: s = sig_h_el(x); break;
            case PGB_XS_H_IONIZE: s = sig_h_ion(x); break;
            case PGB_XS_AR_CX: s = sig_ar_cx(x); break;
            default: s = sig_h_cx(x); break;
        }
        out[k] = (double)s;
    }
}
int pgb_launch_cross_sections(int which, const double* d_e, long long n, double* d_out, cudaStream_t st) {
    k_cross_sections<<<(int)((n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096), 256, 0, st>>>(which, d_e, n, d_out);
    return cudaGetLastError() == cudaSuccess ? 0 : PGB_ERR_CUDA;
}

CollConsts pgb_coll_consts(pgb_run* r) {
    CollConsts c;
    const pgb_params& p = r->p;
    c.species = p.species;
    c.el_const = p.sigma_elastic_mode == PGB_SIGMA_CONSTANT;
    c.ion_const = p.sigma_ionization_mode == PGB_SIGMA_CONSTANT;
    c.cx_const = p.sigma_cx_mode == PGB_SIGMA_CONSTANT;
    c.el_value = (float)p.elastic_sigma_value;
    c.ion_value = (float)p.ionization_sigma_value;
    c.cx_value = (float)p.sigma_value;
    c.e_energy_coef = (float)((0.5 / PGB_CHARGE) * p.electron_mass);
    c.el_max = c.el_const ? c.el_value : (c.species == PGB_ARGON ? 25.5f : 50.5f);
    c.i_energy_coef = (float)((0.5 / PGB_CHARGE) * p.ion_mass);
    c.e_pcoef = (float)(p.dt * 1.0e-20 * p.neutral_density);
    c.i_pcoef = (float)(p.dti * 1.0e-20 * p.neutral_density);
    {
        const double k = (double)c.e_pcoef * (double)c.el_max * 1.000001 * (1.0 + 1.0e-5);
        c.el_bound2 = (float)(k * k * (1.0 + 1.0e-6));
        if (!(c.el_bound2 >= 0.0f)) c.el_bound2 = INFINITY;   /* a negative or NaN bound tests everyone */
    }
    if (c.ion_const) c.ion_emin = c.ion_value > 0.0f ? -INFINITY : INFINITY;
    else c.ion_emin = c.species == PGB_ARGON ? 15.755f : 13.6f;
    c.me = p.electron_mass; c.mi = p.ion_mass; c.dt = p.dt; c.dti = p.dti;
    c.threshold = p.threshold;
    c.reduced_mass = p.ion_mass / (p.electron_mass + p.ion_mass);
    c.n_neutral = p.init_no_neutrals;
    c.seed = p.seed;
    /* (ve + vn) < sqrt(THRESHOLD/rm)/2 makes (rm/2)(ve-vn)^2 at most
     * THRESHOLD/8, far from THRESHOLD whatever the FP32 rounding         */
    {
        double rm = (double)(float)(c.reduced_mass * c.me);
        double cap = 0.5 * sqrt((double)(float)p.threshold / rm) - 1.001 * (double)r->vn_max[0];
        c.ion_vcap = cap > 0.0 ? (float)cap : 0.0f;
    }
    return c;
}

static PushArgs push_args(pgb_run* r, int s) {
    PushArgs a;
    Species& S = r->sp[s];
    a.xv = S.xv; a.vz = S.vz; a.w = S.w; a.id = S.id;
    a.exy = r->exy; a.qacc = r->qacc[s]; a.ds = r->ds; a.s = s;
    a.pc = push_consts(r, s);
    a.cc = pgb_coll_consts(r);
    a.neut = r->neut[0];
    a.pieces = r->pieces[s];
    {
        int nby;
        pgb_bins(r, &a.nbx, &nby);
    }
    a.tl_out = r->tile_list[s == 0 ? LIST_OUT_E : LIST_OUT_I];
    a.tc_out = r->tile_cnt[s == 0 ? LIST_OUT_E : LIST_OUT_I];
    a.tl_ev = r->tile_list[LIST_ION_EV];
    a.tc_ev = r->tile_cnt[LIST_ION_EV];
    return a;
}

/* Whether a push deposits through a window of the whole grid: runs that do
 * not sort (a sorted one's pieces have small windows), on grids of which
 * two windows fit on an SM beside L1 (65 nodes a side), from 16 particles a
 * node.  Both ways add the same integers.  A step of an argon run without
 * sort, straight (deposit_pairs) / window: 17^2 nodes, 1 M particles a
 * species 648 / 54 us; 33^2, 30 K 33 / 33, 300 K 68 / 41; 65^2, 60 K 35 / 35,
 * 150 K 39 / 37, 1 M 91 / 62, 4 M 307 / 163.  129^2, with one window per SM:
 * 300 K 45 / 52, 1 M 83 / 85, 4 M 256 / 243.  The count is the host's latest;
 * it is no part of the result.                                            */
static bool push_whole(const pgb_run* r, int s) {
    const long long nodes = (long long)r->nx * r->ny;
    return r->p.sort_interval == 0 && nodes * 4 <= 48 * 1024 && r->hs->n[s] >= 16 * nodes;
}
int pgb_launch_push(pgb_run* r, int s, bool deposit, bool absorb) {
    PushArgs a = push_args(r, s);
    if (deposit && push_whole(r, s)) {
        void (*kp)(PushArgs) = absorb ? k_push<true, true, true> : k_push<true, false, true>;
        const size_t smem = sizeof(unsigned int) * r->nx * r->ny;
        PGB_CK(r, pgb_launch_pdl(kp, dim3(grid_for(r, 2)), dim3(PGB_PUSH_THREADS), smem, r->stream, a));
    } else {
        void (*kp)(PushArgs) = !deposit ? k_push<false, false, false> : absorb ? k_push<true, true, false> : k_push<true, false, false>;
        PGB_CK(r, pgb_launch_pdl(kp, dim3(grid_for(r, r->tune_push_per_sm)), dim3(PGB_PUSH_THREADS), 0, r->stream, a));
    }
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_flag_outside(pgb_run* r, int s) {
    int l = s == 0 ? LIST_OUT_E : LIST_OUT_I;
    PGB_CK(r, pgb_launch_pdl(k_flag, dim3(grid_for(r, 8)), dim3(PGB_PUSH_THREADS), 0, r->stream, r->sp[s].xv, r->ds, s, r->nx, r->ny, r->ps, r->p.steadystate,
                                                               r->tile_list[l], r->tile_cnt[l]));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}


int pgb_launch_step_advance(pgb_run* r, int commit) {
    PGB_CK(r, pgb_launch_pdl(k_step_advance, dim3(1), dim3(1), 0, r->stream, r->ds, commit));
    r->launches++;
    return 0;
}

/* leave_sms: SMs the collision kernel leaves free (one block fills an SM).
 * Small runs take fewer blocks: one per MCC_GROUPS tiles, from the electron
 * count last read back; the kernel loops over the tiles.                 */
int pgb_launch_mcc(pgb_run* r, int leave_sms, bool count_events) {
    PushArgs a = push_args(r, 0);
    const long long n = std::max<long long>(r->hs->n[0], 0), per = (long long)MCC_GROUPS * PGB_TILE;
    const int g = (int)std::min<long long>(std::max(1, r->sms - leave_sms), std::max<long long>(1, (n + per - 1) / per));
    const size_t smem = sizeof(MccQueue) * MCC_WARPS;
    if (!count_events)   /* the list's counts are added up event by event */
        PGB_CK(r, cudaMemsetAsync(a.tc_ev, 0, sizeof(int) * r->ntiles_cap, r->stream));
    PGB_CK(r, cudaFuncSetAttribute(k_mcc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PGB_CK(r, pgb_launch_pdl(k_mcc, dim3(g), dim3(MCC_THREADS), smem, r->stream, a, count_events ? 0 : 1));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

/* per-tile list `which` (tiles of species s) -> dense list + count */
int pgb_build_list(pgb_run* r, int which, int s, int commit) {
    PGB_CK(r, pgb_launch_pdl(k_build_list, dim3(r->sms), dim3(LIST_THREADS), 0, r->stream, (const int*)r->tile_list[which],
                             (const int*)r->tile_cnt[which], r->ds, s, r->list[which], &r->ds->list_n[which], commit));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_deposit(pgb_run* r, int s) {
    const SlotSource src{r->sp[s].xv, r->sp[s].w};
    const long long n = r->hs->n[s];   /* the host's latest count: it picks the kernel, no result */
    if (deposit_through_windows(n, (long long)r->nx * r->ny)) {
        PGB_CK(r, cudaFuncSetAttribute(k_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DEP_SMEM));
        PGB_CK(r, pgb_launch_pdl(k_deposit, dim3(grid_for(r, DEP_BLOCKS_PER_SM)), dim3(DEP_THREADS), DEP_SMEM, r->stream,
                                 src, r->ds, s, r->nx, r->ny, r->ps, r->qacc[s]));
    } else {
        const long long blocks = std::min<long long>(std::max<long long>((n + 255) / 256, 1), grid_for(r, 8));
        PGB_CK(r, pgb_launch_pdl(k_deposit_few, dim3((unsigned)blocks), dim3(256), 0, r->stream, src, (const DevState*)r->ds,
                                 s, r->nx, r->ny, r->ps, r->qacc[s]));
    }
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_inject(pgb_run* r, int species_mask, bool push_e, int commit, bool absorb_e) {
    InjectArgs a;
    a.e = r->sp[0]; a.i = r->sp[1]; a.ds = r->ds; a.k = r->p.number_to_inject;
    a.dx = r->dx; a.dy = r->dy; a.xlength = r->p.xlength; a.ylength = r->p.ylength;
    a.seed = r->p.seed;
    a.pce = push_consts(r, 0); a.exy = r->exy;
    a.push_e = push_e; a.absorb_e = absorb_e; a.species_mask = species_mask;
    a.list_out_e = r->list[LIST_OUT_E]; a.list_cap = r->list_cap;
    a.flag = r->inject_flag;
    if (a.k <= 0) return 0;
    if (a.k <= INJECT_BLOCK_MAX) {
        const int threads = (a.k + 31) & ~31;
        for (int s = 0; s < 2; ++s)
            if (species_mask & (1 << s)) {
                PGB_CK(r, pgb_launch_pdl(k_inject_block, dim3(1), dim3(threads), 0, r->stream, a, s, commit & (1 << s)));
                r->launches++;
            }
        PGB_CK(r, cudaGetLastError());
        return 0;
    }
    const int tot = a.k * ((species_mask & 1) + ((species_mask >> 1) & 1));
    if (commit) {
        PGB_CK(r, pgb_launch_pdl(k_ionize_count_commit, dim3(1), dim3(1), 0, r->stream, r->ds, commit));
        r->launches++;
    }
    PGB_CK(r, pgb_launch_pdl(k_inject, dim3((tot + 127) / 128), dim3(128), 0, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_inject_commit, dim3(1), dim3(1024), 0, r->stream, a));
    r->launches += 2;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_ionize_appends(pgb_run* r, int store_e, int store_i) {
    IonizeAppendArgs a;
    a.e = r->sp[0]; a.i = r->sp[1]; a.ds = r->ds; a.ev = r->list[LIST_ION_EV];
    a.cc = pgb_coll_consts(r); a.neut = r->neut[0];
    a.dx = r->dx; a.dy = r->dy; a.ps = r->ps;
    a.store_e = store_e;
    a.store_i = store_i;
    PGB_CK(r, pgb_launch_pdl(k_ionize_append, dim3(r->sms * 2), dim3(256), 0, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_ionize_commit, dim3(1), dim3(1), 0, r->stream, r->ds, a.store_e, a.store_i, r->sp[0].cap, r->sp[1].cap));
    r->launches += 2;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_compact(pgb_run* r, int s) {
    Species& S = r->sp[s];
    int* tc = r->tile_cnt[LIST_SPARE];
    int* toff = r->aux_j;
    PGB_CK(r, pgb_launch_pdl(k_alive_count, dim3(grid_for(r, 8)), dim3(PGB_PUSH_THREADS), 0, r->stream, S.xv, r->ds, s, tc));
    r->launches++;
    PGB_CK(r, pgb_launch_pdl(k_scan_small, dim3(1), dim3(1024), 0, r->stream, tc, toff, &r->ds->n[s], 0, &r->ds->list_n[LIST_SPARE]));
    r->launches++;
    PGB_CK(r, pgb_launch_pdl(k_compact, dim3(grid_for(r, 8)), dim3(PGB_PUSH_THREADS), 0, r->stream, S, r->ds, s, toff));
    r->launches++;
    PGB_CK(r, pgb_launch_pdl(k_compact_commit, dim3(1), dim3(1), 0, r->stream, r->ds, s, &r->ds->list_n[LIST_SPARE]));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    std::swap(S.xv, S.xv2);
    std::swap(S.vz, S.vz2);
    std::swap(S.w, S.w2);
    std::swap(S.id, S.id2);
    return 0;
}

int pgb_launch_load(pgb_run* r, int s, const double* d_aos, long long i0, long long i1) {
    PGB_CK(r, pgb_launch_pdl(k_load, dim3(grid_for(r, 4)), dim3(256), 0, r->stream, r->sp[s], d_aos, i0, i1, r->dx, r->dy,
                             pgb_pos_scale(r->dx, r->ps), pgb_pos_scale(r->dy, r->ps), r->ps));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_load_commit(pgb_run* r, int s, long long n) {
    PGB_CK(r, pgb_launch_pdl(k_load_commit, dim3(1), dim3(1), 0, r->stream, r->ds, s, n));
    r->launches++;
    return 0;
}
int pgb_launch_set_step(pgb_run* r, long long t, double phi, bool one) {
    PGB_CK(r, pgb_launch_pdl(k_set_step, dim3(1), dim3(1), 0, r->stream, r->ds, t, r->phi_tab, phi, one ? 1 : 0));
    r->launches++;
    return 0;
}

/* live-slot offsets per tile (into r->aux_j) for pgb_launch_dump */
int pgb_launch_dump_offsets(pgb_run* r, int s) {
    int* tc = r->tile_cnt[LIST_SPARE];
    PGB_CK(r, pgb_launch_pdl(k_alive_count, dim3(grid_for(r, 8)), dim3(PGB_PUSH_THREADS), 0, r->stream, r->sp[s].xv, r->ds, s, tc));
    r->launches++;
    PGB_CK(r, pgb_launch_pdl(k_scan_small, dim3(1), dim3(1024), 0, r->stream, tc, r->aux_j, &r->ds->n[s], 0, &r->ds->list_n[LIST_SPARE]));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

int pgb_launch_dump(pgb_run* r, int s, double* d_out, unsigned int* d_ids, long long cap, int t0, int t1) {
    PGB_CK(r, pgb_launch_pdl(k_dump, dim3(grid_for(r, 8)), dim3(PGB_PUSH_THREADS), 0, r->stream, r->sp[s], r->ds, s, (const int*)r->aux_j, ldexp(r->dx, -r->ps),
                             ldexp(r->dy, -r->ps), d_out, d_ids, cap, t0, t1));
    r->launches++;
    PGB_CK(r, cudaGetLastError());
    return 0;
}

