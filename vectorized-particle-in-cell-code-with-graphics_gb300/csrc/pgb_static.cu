/*
 * pgb_deposit_static: the charge deposit of one species without a run handle
 * and without allocating device memory.
 *
 * Callers that can't allocate:
 *   - a diagnostic or viewer hook that runs between steps on the
 *     simulation's own stream, with the particles already on the device.
 *     cudaMalloc and cudaFree synchronise the whole device, which would drain
 *     the step queue the caller keeps full;
 *   - a host that has reserved the device memory for particle capacity.
 *     There, a temporary grid-sized allocation can fail in the middle of a
 *     run.
 *
 * Output: the same grid as pgb_deposit + pgb_get_grid(PGB_GRID_Q_E/Q_I) for
 * the same particle records.  That is particle::collect_charge:
 *   - CIC weights (pic.cl:22-52);
 *   - the charge density qc/(DX*DY);
 *   - edge rows and columns doubled, corners doubled again
 *     (particle.cpp:663-858).
 * The per-node sums are int64 fixed point (2^19 per unit weight), so the
 * grid does not depend on the order of the records.
 *
 * Scratch: one int64 accumulator per node.  It lives in the file-scope
 * array g_static_acc below, of PGB_STATIC_DEPOSIT_MAX_NODES entries
 * (513 x 513 nodes, 2.1 MB), so no call allocates.  The rules that follow:
 *   - Every call shares the array and leaves its own sums in it.  Each call
 *     clears the nodes it uses before depositing.
 *   - Two calls whose kernels overlap on the GPU race on the array, for
 *     example calls on two streams without an event between them.  Calls on
 *     one stream are ordered and safe.
 *   - The first call on a device, with that device current, finds the
 *     array's address with cudaGetSymbolAddress and caches it.  This loads
 *     the module on that device if it is not loaded yet.  Make that first
 *     call before any stream capture begins.
 *   - The cached address belongs to the device's primary context.  After
 *     cudaDeviceReset on a device the module may load elsewhere, so the
 *     entry point must not be called on that device again in this process.
 */
#include <cuda_runtime.h>
#include <mutex>
#include <string>
#include "pgb_internal.h"
#include "pgb_physics.cuh"
#include "pgb_deposit.cuh"

#define PGB_STATIC_MAX_DEVICES 64

/* the shared accumulator: [ny][nx] int64 fixed point, nx*ny <= maximum */
static __device__ __align__(256) unsigned long long g_static_acc[PGB_STATIC_DEPOSIT_MAX_NODES];

namespace {

struct DeviceSetup {
    unsigned long long* acc = nullptr;   /* device address of g_static_acc */
    int sms = 0;
};

std::mutex g_setup_mu;
DeviceSetup g_setup[PGB_STATIC_MAX_DEVICES];

__global__ void k_static_clear(unsigned long long* acc, int nodes) {
    pgb_pdl_entry();
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nodes; k += gridDim.x * blockDim.x) acc[k] = 0ull;
}

/* Each record is a particleVec {x, y, vx, vy, vz, w} (particleVec.h:26-35).
 * x and y become fixed-point positions exactly as pgb_load_species makes
 * them (pgb_pos_shift of the grid), so the deposit is bit-identical to the
 * run handle's.                                                          */
struct RecordSource {
    const double* aos6;
    double dx, dy;
    PosScale rx, ry;
    int ps;
    __device__ __forceinline__ void operator()(long long i, float& x, float& y, float& w) const {
        const double* const r = aos6 + 6 * i;
        x = pos_from_m(r[0], dx, rx, ps);
        y = pos_from_m(r[1], dy, ry, ps);
        w = weight_from_double(r[5]);
    }
};
/* few records for the grid: one thread each, straight to the accumulator */
__global__ void __launch_bounds__(256) k_static_deposit_few(RecordSource src, long long n, int nx, int ny,
                                                            unsigned long long* acc) {
    pgb_pdl_entry();
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    float x = pos_dead(), y = pos_dead(), w = 0.0f;
    if (i < n) src(i, x, y, w);
    deposit_pairs(acc, nx, src.ps, deposit_ok(x, y, nx, ny, src.ps), x, y, w);
}
__global__ void __launch_bounds__(DEP_THREADS) k_static_deposit(RecordSource src, long long n, int nx, int ny,
                                                                unsigned long long* acc) {
    pgb_pdl_entry();
    deposit_windows(src, n, nx, ny, src.ps, acc);
}

/* q = (sum / PGB_FIX_SCALE * qc/(DX*DY)) * edge factor, the sum being in
 * units of 2^-19 of a unit weight (particle.cpp:829-845)                  */
__global__ void k_static_finish(const unsigned long long* acc, int nx, int ny, double qcdxdy, double* q) {
    pgb_pdl_entry();
    const int nodes = nx * ny;
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nodes; k += gridDim.x * blockDim.x) {
        int j = k / nx, i = k - j * nx;
        bool ex = (i == 0 || i == nx - 1), ey = (j == 0 || j == ny - 1);
        double ef = (ex ? 2.0 : 1.0) * (ey ? 2.0 : 1.0) * ((ex && ey) ? 2.0 : 1.0);
        double v = __dmul_rn((double)(long long)acc[k], 1.0 / PGB_FIX_SCALE);
        q[k] = __dmul_rn(__dmul_rn(v, qcdxdy), ef);
    }
}

int setup_error(const std::string& msg, cudaError_t e) {
    pgb_set_unbound_error(msg + ": " + cudaGetErrorString(e));
    return PGB_ERR_CUDA;
}

/* per-device set-up, once per device, with that device current */
int device_setup(DeviceSetup* out) {
    int dev = -1;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return setup_error("pgb_deposit_static: cudaGetDevice", e);
    if (dev < 0 || dev >= PGB_STATIC_MAX_DEVICES) {
        pgb_set_unbound_error("pgb_deposit_static: device ordinal " + std::to_string(dev) + " is beyond " +
                              std::to_string(PGB_STATIC_MAX_DEVICES));
        return PGB_ERR_ARG;
    }
    std::lock_guard<std::mutex> lock(g_setup_mu);
    DeviceSetup& s = g_setup[dev];
    if (!s.acc) {
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_static_acc);
        if (e != cudaSuccess) return setup_error("pgb_deposit_static: cudaGetSymbolAddress", e);
        int sms = 0;
        e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return setup_error("pgb_deposit_static: cudaDeviceGetAttribute", e);
        s.sms = sms > 0 ? sms : 1;
        s.acc = (unsigned long long*)p;
    }
    *out = s;
    return 0;
}

}  // namespace

extern "C" int pgb_deposit_static(const double* d_aos6, int64_t n, int32_t nx, int32_t ny, double dx, double dy,
                                  double qc, double* d_q, void* stream) {
    if (n < 0 || (n > 0 && !d_aos6) || !d_q || nx < 2 || ny < 2 || !(dx > 0.0) || !(dy > 0.0)) {
        pgb_set_unbound_error("pgb_deposit_static: bad argument");
        return PGB_ERR_ARG;
    }
    if ((int64_t)nx * ny > PGB_STATIC_DEPOSIT_MAX_NODES) {
        pgb_set_unbound_error("pgb_deposit_static: grid of " + std::to_string(nx) + " x " + std::to_string(ny) +
                              " nodes exceeds the static scratch maximum of " +
                              std::to_string(PGB_STATIC_DEPOSIT_MAX_NODES) + " nodes (513 x 513)");
        return PGB_ERR_CAPACITY;
    }
    DeviceSetup s;
    int rc = device_setup(&s);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    const int nodes = nx * ny;
    const int gblocks = (nodes + 255) / 256 < s.sms * 4 ? (nodes + 255) / 256 : s.sms * 4;
    const int ps = pgb_pos_shift(nx, ny);
    const RecordSource src{d_aos6, dx, dy, pgb_pos_scale(dx, ps), pgb_pos_scale(dy, ps), ps};
    cudaError_t e = pgb_launch_pdl(k_static_clear, dim3(gblocks), dim3(256), 0, st, s.acc, nodes);
    if (e != cudaSuccess) return setup_error("pgb_deposit_static: kernel launch", e);
    if (deposit_through_windows(n, nodes)) {
        /* a block's window is zeroed and flushed once per run of records */
        const long long want = (n + DEP_CHUNK - 1) / DEP_CHUNK;
        const int blocks = want < (long long)s.sms * DEP_BLOCKS_PER_SM ? (int)want : s.sms * DEP_BLOCKS_PER_SM;
        e = cudaFuncSetAttribute(k_static_deposit, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DEP_SMEM);
        if (e == cudaSuccess)
            e = pgb_launch_pdl(k_static_deposit, dim3(blocks), dim3(DEP_THREADS), DEP_SMEM, st, src, (long long)n, nx, ny, s.acc);
    } else if (n > 0) {
        e = pgb_launch_pdl(k_static_deposit_few, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, st, src, (long long)n, nx, ny, s.acc);
    }
    if (e == cudaSuccess)
        e = pgb_launch_pdl(k_static_finish, dim3(gblocks), dim3(256), 0, st, (const unsigned long long*)s.acc, nx, ny,
                           qc / (dx * dy), d_q);
    if (e != cudaSuccess) return setup_error("pgb_deposit_static: kernel launch", e);
    e = cudaGetLastError();
    if (e != cudaSuccess) return setup_error("pgb_deposit_static: kernel launch", e);
    return 0;
}
