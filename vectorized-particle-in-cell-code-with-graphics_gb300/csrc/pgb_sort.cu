/*
 * Spatial binning of the particles (stable counting sort by bin).
 *
 * The deposit (particle::collect_charge, pic.cl:22-52) scatters four adds
 * per particle; on particles in arbitrary order they land on random grid
 * nodes and the adds go to L2 as global atomics.  Every sort_interval steps
 * the particles of a species are re-ordered by bin (BIN x BIN cells), each
 * bin starting on a 1024-slot tile boundary, so the push kernel can give a
 * CTA a run of tiles of one bin and accumulate its deposit in a shared-
 * memory window of the bin's nodes plus a halo.
 *
 * The sort is stable (particles keep their relative order within a bin),
 * so the resulting order -- and every order-dependent rule that follows it
 * (charge-exchange accumulation, wall-list order) -- is deterministic.  It
 * also drops removed particles (tombstones).  Passes:
 *   count    per chunk of SORT_CHUNK slots, a shared histogram of bin keys
 *   scan     per bin over chunks, then over bins with tile padding (and the
 *            work pieces: runs of tiles of one bin)
 *   scatter  one CTA per chunk sorts it in shared memory and writes each
 *            bin's run of particles to its place
 * Bound by memory traffic: 16 B read by the count, 28 B read and written
 * by the scatter per particle.  A warp that placed its particles straight
 * from registers wrote them a few at a time (half a sector of 32 B per
 * position, an eighth per vz, weight and id): 1.2 ms for 16 Mi particles
 * loaded in random order.  Sorted in shared memory first, a chunk of 4096
 * over 257 bins leaves in runs of 16 particles.
 */
#include <cuda_runtime.h>
#include "pgb_internal.h"
#include "pgb_physics.cuh"

#define SORT_CHUNK PGB_SORT_CHUNK

struct SortArgs {
    Species S;
    DevState* ds;
    int s;
    int nx, ny;              /* nodes */
    int ps;                  /* fraction bits of the positions */
    int nbx, nby, nbins;     /* bins; key nbins = not in the deposit region */
    int* counts;             /* [chunk][key] */
    int* offs;               /* [chunk][key] exclusive within the key */
    int* key_total;          /* [key] */
    long long* key_start;    /* [key+1] padded starts */
    int4* pieces;            /* {first tile, tiles, bin, 0} */
    int want_pieces;         /* pieces that keep the push's grid busy */
};

__device__ __forceinline__ int bin_key(float4 p, int nx, int ny, int ps, int nbx, int nbins) {
    if (is_dead(p.x)) return -1;
    int jp = pcell(p.x, ps), kp = pcell(p.y, ps);
    /* the deposit region of collectCharge (pic.cl:35) */
    if (!deposit_ok(p.x, p.y, nx, ny, ps)) return nbins;
    return (kp / PGB_BIN) * nbx + (jp / PGB_BIN);
}

__global__ void __launch_bounds__(512) k_sort_count(SortArgs a) {
    pgb_pdl_entry();
    extern __shared__ int s_hist[];
    const long long n = a.ds->n[a.s];
    const int nch = (int)((n + SORT_CHUNK - 1) / SORT_CHUNK);
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        for (int k = threadIdx.x; k <= a.nbins; k += blockDim.x) s_hist[k] = 0;
        __syncthreads();
        float4 p[SORT_CHUNK / 512];
#pragma unroll
        for (int q = 0; q < SORT_CHUNK / 512; ++q) {
            const long long i = (long long)c * SORT_CHUNK + q * 512 + threadIdx.x;
            p[q] = i < n ? a.S.xv[i] : make_float4(pos_dead(), 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int q = 0; q < SORT_CHUNK / 512; ++q) {
            const int key = bin_key(p[q], a.nx, a.ny, a.ps, a.nbx, a.nbins);
            if (key >= 0) atomicAdd(&s_hist[key], 1);
        }
        __syncthreads();
        for (int k = threadIdx.x; k <= a.nbins; k += blockDim.x) a.counts[(long long)c * (a.nbins + 1) + k] = s_hist[k];
        __syncthreads();
    }
}

/* exclusive scan of one value per thread over the CTA; *total = the sum.
 * Every thread of the CTA must call it.                                  */
__device__ __forceinline__ long long block_excl_scan_ll(long long v, long long* s_w, long long& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    long long x = v;
    for (int d = 1; d < 32; d <<= 1) {
        long long y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_w[warp] = x;
    __syncthreads();
    if (warp == 0) {
        long long w = lane < nw ? s_w[lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            long long y = __shfl_up_sync(0xffffffffu, w, d);
            if (lane >= d) w += y;
        }
        if (lane < nw) s_w[lane] = w;   /* inclusive over warps */
    }
    __syncthreads();
    long long before = warp ? s_w[warp - 1] : 0;
    total = s_w[nw - 1];
    __syncthreads();
    return before + x - v;
}

/* per key: exclusive scan over the chunks.  A CTA takes eight keys (a
 * sector of each chunk's row) and splits the chunks into 128 runs, a run and
 * key per thread: sums, a warp's scan over the runs per key, offsets.  (With
 * 32 keys and 32 runs per CTA the 257 keys of 513^2 were 9 CTAs: 30 us for
 * 16 Mi particles, now 15.)                                              */
#define SCAN_KEYS 8
#define SCAN_RUNS 128
__global__ void __launch_bounds__(SCAN_KEYS * SCAN_RUNS) k_sort_scan_keys(SortArgs a) {
    pgb_pdl_entry();
    __shared__ int s_sum[SCAN_KEYS][SCAN_RUNS + 1];
    const long long n = a.ds->n[a.s];
    const int nch = (int)((n + SORT_CHUNK - 1) / SORT_CHUNK), nk = a.nbins + 1;
    const int sub = threadIdx.x % SCAN_KEYS, run = threadIdx.x / SCAN_KEYS;
    const int key = blockIdx.x * SCAN_KEYS + sub;
    const int per = (nch + SCAN_RUNS - 1) / SCAN_RUNS, c0 = min(run * per, nch), c1 = min(c0 + per, nch);
    int sum = 0;
    if (key < nk) {
#pragma unroll 8
        for (int c = c0; c < c1; ++c) sum += a.counts[(long long)c * nk + key];
    }
    s_sum[sub][run] = sum;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < SCAN_KEYS) {
        int* const v = s_sum[warp] + lane * (SCAN_RUNS / 32);
        int t = 0;
#pragma unroll
        for (int q = 0; q < SCAN_RUNS / 32; ++q) t += v[q];
        int x = t;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        const int k = blockIdx.x * SCAN_KEYS + warp;
        if (lane == 31 && k < nk) a.key_total[k] = x;
        x -= t;
#pragma unroll
        for (int q = 0; q < SCAN_RUNS / 32; ++q) {
            const int c = v[q];
            v[q] = x;
            x += c;
        }
    }
    __syncthreads();
    if (key >= nk) return;
    int acc = s_sum[sub][run];
#pragma unroll 8
    for (int c = c0; c < c1; ++c) {
        const int v = a.counts[(long long)c * nk + key];
        a.offs[(long long)c * nk + key] = acc;
        acc += v;
    }
}

/* over keys: padded starts (each key begins on a tile boundary), pieces.
 * One CTA scans the keys 1024 at a time (tiles and pieces per key) and
 * each key's thread writes its pieces.                                   */
__global__ void __launch_bounds__(1024) k_sort_scan_bins(SortArgs a) {
    pgb_pdl_entry();
    __shared__ long long s_w[32];
    long long carry_t = 0, carry_p = 0, live = 0;
    /* A piece is a run of tiles of one bin that one CTA of the push takes:
     * PGB_PIECE_TILES tiles (what its window's 32-bit sums allow), fewer
     * where that would leave CTAs idle: 200k particles at 65^2 nodes are 49
     * pieces of four tiles, and the electron push took 17 us on 49 SMs.     */
    long long tiles_all = 0;
    for (int base = 0; base <= a.nbins; base += blockDim.x) {
        const int key = base + threadIdx.x;
        const long long tiles = key <= a.nbins ? (a.key_total[key] + PGB_TILE - 1) / PGB_TILE : 0;
        long long tot;
        (void)block_excl_scan_ll(tiles, s_w, tot);
        tiles_all += tot;
    }
    const long long piece_tiles = min((long long)PGB_PIECE_TILES, max(1ll, tiles_all / a.want_pieces));
    for (int base = 0; base <= a.nbins; base += blockDim.x) {
        const int key = base + threadIdx.x;
        long long tiles = 0, np = 0, c = 0;
        if (key <= a.nbins) {
            c = a.key_total[key];
            tiles = (c + PGB_TILE - 1) / PGB_TILE;
            np = (tiles + piece_tiles - 1) / piece_tiles;
        }
        long long tot_t, tot_p, tot_c;
        (void)block_excl_scan_ll(c, s_w, tot_c);
        live += tot_c;
        long long t0 = carry_t + block_excl_scan_ll(tiles, s_w, tot_t);
        long long p0 = carry_p + block_excl_scan_ll(np, s_w, tot_p);
        if (key <= a.nbins) {
            a.key_start[key] = t0 * PGB_TILE;
            const int bin = key < a.nbins ? key : -1;
            for (long long q = 0; q < np; ++q) {
                long long t = q * piece_tiles;
                int len = (int)((tiles - t) < piece_tiles ? (tiles - t) : piece_tiles);
                a.pieces[p0 + q] = make_int4((int)(t0 + t), len, bin, 0);
            }
        }
        carry_t += tot_t;
        carry_p += tot_p;
    }
    /* every bin starts on a tile boundary: the padded layout needs carry_t
     * tiles.  If they do not fit the capacity, the sort copies the
     * particles in their current order instead (no pieces, no padding) and
     * the step reports the capacity error.                              */
    if (threadIdx.x == 0) {
        const int over = carry_t * PGB_TILE > a.S.cap ? 1 : 0;
        a.ds->sort_overflow = over;
        a.ds->list_n[LIST_SPARE] = live;
        a.key_start[a.nbins + 1] = carry_t * PGB_TILE;
        a.ds->n_pieces[a.s] = over ? 0 : (int)carry_p;
        a.ds->sorted_tiles[a.s] = over ? 0 : carry_t;
        if (over) atomicOr(&a.ds->err, a.s == 0 ? ERR_CAP_E : ERR_CAP_I);
    }
}

/* One CTA per chunk of SORT_CHUNK slots.  A warp takes 256 consecutive
 * slots, 32 at a time: a particle's rank within its warp is the warp's
 * running count of its key plus the lanes of the same key before it; the
 * warps' counts are then scanned per key and the keys over the chunk, which
 * gives each particle its place in the sorted chunk.  The particles go
 * there in shared memory and leave from there, bin after bin.
 * What bounds it is the latency of shared memory (the counts are a chain
 * from item to item) and of the loads, so two CTAs share an SM: at 123
 * registers a thread one filled it, and a 16 Mi sort's scatter took 313 us,
 * now 224 (0.94 GB, 4.2 TB/s).                                           */
#define SORT_THREADS 512
#define SORT_WARPS (SORT_THREADS / 32)
#define SORT_ITEMS (SORT_CHUNK / SORT_THREADS)
static_assert(SORT_CHUNK <= 65536, "ranks within a chunk are 16 bits");
/* dynamic shared memory: the staged particles, their keys, the counts per
 * warp and key, the destination of each key's run                        */
static size_t sort_smem(int nkeys) {
    const size_t w = ((size_t)nkeys * SORT_WARPS * sizeof(unsigned short) + 15) & ~(size_t)15;
    return SORT_CHUNK * (sizeof(float4) + sizeof(unsigned short)) + w + (size_t)nkeys * sizeof(long long);
}
__global__ void __launch_bounds__(SORT_THREADS, 2) k_sort_scatter(SortArgs a) {
    pgb_pdl_entry();
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int nk = a.nbins + 1;
    float4* const s_xv = reinterpret_cast<float4*>(s_raw);
    unsigned short* const s_key = reinterpret_cast<unsigned short*>(s_raw + SORT_CHUNK * sizeof(float4));
    unsigned short* const s_cnt = s_key + SORT_CHUNK;   /* [warp][key] */
    long long* const s_dst = reinterpret_cast<long long*>(
        s_raw + SORT_CHUNK * (sizeof(float4) + sizeof(unsigned short)) +
        (((size_t)nk * SORT_WARPS * sizeof(unsigned short) + 15) & ~(size_t)15));
    __shared__ int s_w[SORT_WARPS];
    const long long n = a.ds->n[a.s];
    const int nch = (int)((n + SORT_CHUNK - 1) / SORT_CHUNK);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    if (a.ds->sort_overflow) {
        /* the padded layout does not fit: keep the order (and the slots) */
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
            a.S.xv2[i] = a.S.xv[i];
            a.S.vz2[i] = a.S.vz[i];
            a.S.w2[i] = a.S.w[i];
            a.S.id2[i] = a.S.id[i];
        }
        return;
    }
    for (int c = blockIdx.x; c < nch; c += gridDim.x) {
        const long long base = (long long)c * SORT_CHUNK + warp * (32 * SORT_ITEMS) + lane;
        float4 p[SORT_ITEMS];
#pragma unroll
        for (int q = 0; q < SORT_ITEMS; ++q) {
            const long long i = base + 32 * q;
            p[q] = i < n ? a.S.xv[i] : make_float4(pos_dead(), 0.f, 0.f, 0.f);
        }
        for (int k = threadIdx.x; k < nk * SORT_WARPS; k += SORT_THREADS) s_cnt[k] = 0;
        __syncthreads();
        int key[SORT_ITEMS], pos[SORT_ITEMS];
        unsigned short* const cnt = s_cnt + warp * nk;
#pragma unroll
        for (int q = 0; q < SORT_ITEMS; ++q) {
            key[q] = bin_key(p[q], a.nx, a.ny, a.ps, a.nbx, a.nbins);
            const unsigned peers = __match_any_sync(0xffffffffu, key[q]);
            pos[q] = key[q] >= 0 ? cnt[key[q]] + __popc(peers & lt) : -1;
            __syncwarp();
            if (key[q] >= 0 && (peers & lt) == 0) cnt[key[q]] = (unsigned short)(cnt[key[q]] + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        /* per key: exclusive over the warps; over the keys: exclusive */
        int carry = 0;
        for (int b = 0; b < nk; b += SORT_THREADS) {
            const int k = b + threadIdx.x;
            int tot = 0;
            if (k < nk) {
#pragma unroll
                for (int w = 0; w < SORT_WARPS; ++w) tot += s_cnt[w * nk + k];
            }
            int x = tot;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d) x += y;
            }
            if (lane == 31) s_w[warp] = x;
            __syncthreads();
            int before = 0, all = 0;
#pragma unroll
            for (int w = 0; w < SORT_WARPS; ++w) {
                if (w < warp) before += s_w[w];
                all += s_w[w];
            }
            const int start = carry + before + x - tot;   /* of key k in the sorted chunk */
            if (k < nk) {
                int acc = start;
#pragma unroll
                for (int w = 0; w < SORT_WARPS; ++w) {
                    const int v = s_cnt[w * nk + k];
                    s_cnt[w * nk + k] = (unsigned short)acc;
                    acc += v;
                }
                s_dst[k] = a.key_start[k] + a.offs[(long long)c * nk + k] - start;
            }
            carry += all;
            __syncthreads();
        }
        /* positions and in-plane velocities */
#pragma unroll
        for (int q = 0; q < SORT_ITEMS; ++q)
            if (pos[q] >= 0) {
                pos[q] += cnt[key[q]];
                s_xv[pos[q]] = p[q];
                s_key[pos[q]] = (unsigned short)key[q];
            }
        float vz[SORT_ITEMS], wt[SORT_ITEMS];
        unsigned int id[SORT_ITEMS];
#pragma unroll
        for (int q = 0; q < SORT_ITEMS; ++q) {
            const long long i = base + 32 * q;
            vz[q] = wt[q] = 0.f;
            id[q] = 0u;
            if (pos[q] >= 0) {
                vz[q] = a.S.vz[i];
                wt[q] = a.S.w[i];
                id[q] = a.S.id[i];
            }
        }
        __syncthreads();
        for (int j = threadIdx.x; j < carry; j += SORT_THREADS) {
            const long long d = j + s_dst[s_key[j]];
            if (d < a.S.cap) a.S.xv2[d] = s_xv[j];
        }
        __syncthreads();
        /* the other three arrays in the same space */
        float* const s_vz = reinterpret_cast<float*>(s_raw);
        float* const s_wt = s_vz + SORT_CHUNK;
        unsigned int* const s_id = reinterpret_cast<unsigned int*>(s_wt + SORT_CHUNK);
#pragma unroll
        for (int q = 0; q < SORT_ITEMS; ++q)
            if (pos[q] >= 0) {
                s_vz[pos[q]] = vz[q];
                s_wt[pos[q]] = wt[q];
                s_id[pos[q]] = id[q];
            }
        __syncthreads();
        for (int j = threadIdx.x; j < carry; j += SORT_THREADS) {
            const long long d = j + s_dst[s_key[j]];
            if (d < a.S.cap) {
                a.S.vz2[d] = s_vz[j];
                a.S.w2[d] = s_wt[j];
                a.S.id2[d] = s_id[j];
            }
        }
        __syncthreads();
    }
}

/* tombstones in the padding after each key's particles; new counts */
__global__ void k_sort_pad(SortArgs a) {
    pgb_pdl_entry();
    if (a.ds->sort_overflow) return;   /* the copy kept n and the tombstones */
    for (int key = blockIdx.x; key <= a.nbins; key += gridDim.x) {
        long long s0 = a.key_start[key] + a.key_total[key], s1 = a.key_start[key + 1];
        for (long long i = s0 + threadIdx.x; i < s1; i += blockDim.x) {
            a.S.xv2[i] = make_float4(pos_dead(), 0.f, 0.f, 0.f);
            a.S.vz2[i] = 0.f;
            a.S.w2[i] = 0.f;
            a.S.id2[i] = 0u;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const long long live = a.ds->list_n[LIST_SPARE];
        long long tot = a.key_start[a.nbins + 1];
        a.ds->n[a.s] = tot;
        a.ds->dead[a.s] = tot - live;
    }
}

/* ============================================================ host side */
void pgb_bins(pgb_run* r, int* nbx, int* nby) {
    *nbx = (r->nx - 1 + PGB_BIN - 1) / PGB_BIN;
    *nby = (r->ny - 1 + PGB_BIN - 1) / PGB_BIN;
}

int pgb_launch_sort(pgb_run* r, int s) {
    SortArgs a;
    a.S = r->sp[s]; a.ds = r->ds; a.s = s; a.nx = r->nx; a.ny = r->ny; a.ps = r->ps;
    pgb_bins(r, &a.nbx, &a.nby);
    a.nbins = a.nbx * a.nby;
    a.counts = r->sort_counts; a.offs = r->sort_offs; a.key_total = r->sort_key_total;
    a.key_start = r->sort_key_start; a.pieces = r->pieces[s];
    a.want_pieces = 2 * r->sms;
    const int nk = a.nbins + 1;
    PGB_CK(r, pgb_launch_pdl(k_sort_count, dim3(r->sms * 4), dim3(512), sizeof(int) * nk, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_sort_scan_keys, dim3((nk + SCAN_KEYS - 1) / SCAN_KEYS), dim3(SCAN_KEYS * SCAN_RUNS), 0, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_sort_scan_bins, dim3(1), dim3(1024), 0, r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_sort_scatter, dim3(r->sms * 2), dim3(SORT_THREADS), sort_smem(nk), r->stream, a));
    PGB_CK(r, pgb_launch_pdl(k_sort_pad, dim3(r->sms), dim3(256), 0, r->stream, a));
    r->launches += 5;
    PGB_CK(r, cudaGetLastError());
    Species& S = r->sp[s];
    std::swap(S.xv, S.xv2);
    std::swap(S.vz, S.vz2);
    std::swap(S.w, S.w2);
    std::swap(S.id, S.id2);
    return 0;
}

int pgb_sort_setup(pgb_run* r) {
    int nbx, nby;
    pgb_bins(r, &nbx, &nby);
    const int nk = nbx * nby + 1;
    /* the limit belongs to the kernel, which runs of every grid share: it is
     * set to the most any of them may ask for (a grid that asks for more is
     * refused here)                                                       */
    const size_t most = 224 * 1024;
    PGB_CK(r, cudaFuncSetAttribute(k_sort_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(sort_smem(nk) > most ? sort_smem(nk) : most)));
    size_t hist = sizeof(int) * nk;
    if (hist > 48 * 1024) PGB_CK(r, cudaFuncSetAttribute(k_sort_count, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)hist));
    return 0;
}
