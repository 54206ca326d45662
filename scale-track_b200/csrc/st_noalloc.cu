/*
 * st_noalloc.cu -- st_step_noalloc: one mixed-precision parcel step that allocates nothing.
 *
 * Some callers cannot call cudaMalloc: a host application that hands all device memory to
 * its own pool allocator, code running under a memory budget enforced by a framework, or a
 * plugin that must not grow the process's device footprint after set-up.  For them this
 * entry point runs the same step kernel as st_step on caller-owned parcel, fluid and source
 * arrays, and keeps its only scratch -- the fixed-point source accumulator and a control
 * block -- in a file-scope device array of fixed size.  It calls no cudaMalloc, cudaFree
 * or allocating library routine.
 *
 * The scratch array lives in every GPU that loads this library until the process exits.
 * Its device address is looked up once per device, on the first call made on that device
 * (cudaGetSymbolAddress with that device current), and kept for the life of the process: a
 * cudaDeviceReset of that device makes the kept address stale, so the entry point must not
 * be called on a device after it was reset.  Every call ends by reading the control block
 * back and synchronising the stream, so a call cannot be recorded into a CUDA graph: one
 * made on a capturing stream is rejected before anything is launched.  All calls share the
 * one array and it keeps the last call's contents: each call clears the accumulator before
 * use and resets the control blocks of the call after it (st_turns.h), and calls that overlap on
 * the GPU (other streams or host threads) race on the array; calls after them are sound again.
 */
#include <algorithm>
#include <climits>
#include <cstdint>
#include <mutex>

#include <cuda_runtime.h>

#include "scaletrack.h"
#include "st_device.cuh"
#include "st_turns.h"

using namespace st;

namespace {

constexpr int64_t NOALLOC_MAX_CELLS = ST_NOALLOC_MAX_CELLS;  /* include/scaletrack.h */
/* the accumulator */
static __device__ unsigned long long g_st_noalloc_acc[NOALLOC_MAX_CELLS * 3];

/* Control blocks of the probe and the step, two sets used in turn: every call's last kernel
 * resets the set of the next call (st_turns.h). */
struct CtlPair {
    CloudCtl probe, step;
};
#define ST_CTL0 {0, EXP_NONE, 0, 0, 0ULL, 0ULL}
static __device__ CtlPair g_st_noalloc_ctl[2] = {{ST_CTL0, ST_CTL0}, {ST_CTL0, ST_CTL0}};
#undef ST_CTL0

constexpr int MAX_DEVICES = 64;
struct Scratch {
    CtlPair* ctl = nullptr;
    unsigned long long* acc = nullptr;
    int resident[2] = {0, 0};  /* step blocks that stay resident on the device: one substep, several */
    Turns turns;
};
std::mutex g_mu;
Scratch g_scratch[MAX_DEVICES];

/* One call's turn with the control sets of a device. */
struct Call {
    int dev;
    Turns::Turn turn;
    cudaStream_t s;
    bool complete = false;   /* every kernel of the call has run */
    Call(int device, const Turns::Turn& t, cudaStream_t stream) : dev(device), turn(t), s(stream) {}
    Call(const Call&) = delete;
    ~Call()
    {
        if (!complete) cudaStreamSynchronize(s);   /* what was launched before the failure */
        std::lock_guard<std::mutex> lk(g_mu);
        g_scratch[dev].turns.end(complete);
    }
};

int fail(int code, const char* msg)
{
    st_set_last_error(msg);
    return code;
}

__device__ __forceinline__ void reset(CtlPair* c)
{
    const CloudCtl c0 = {0, EXP_NONE, 0, 0, 0ULL, 0ULL};
    c->probe = c0;
    c->step = c0;
}

__global__ void k_noalloc_reset(CtlPair* both)
{
    if (threadIdx.x < 2) reset(both + threadIdx.x);
}

/* Fixed point -> FP64 into the caller's [nCells][3] source (any length, scalar stores), and
 * the control set of the next call.
 *
 * A call is a chain of three kernels, each launched programmatically behind the one before
 * (its launch and set-up overlap the previous kernel's end): the probe, which also clears the
 * accumulator; the step, its scale straight from the probe's control block; the conversion.
 * What bounds the smallest calls is the chain's latency and the read-back of the control block:
 * 3001 parcels on 12^3 cells took 48.8 us as a memset and five kernels in stream order with the
 * occupancy queried on every call, 32.0 us now (a kernel and a read-back alone: 20 us); 1e6 on
 * 64^3 cells 87.6 -> 78.4 us.
 *
 * acc: plain loads.  The blocks of this kernel may be resident while the probe still clears the
 * accumulator and the step adds to it, so it is not read-only for the kernel's lifetime, as
 * const __restrict__ or __ldg would promise. */
__global__ void __launch_bounds__(256) k_noalloc_finalize(
    const unsigned long long* acc, const CtlPair* ctl, CtlPair* next, int H, double* src,
    int64_t ncomp)
{
    grid_dep_wait();
    if (blockIdx.x == 0 && threadIdx.x == 0) reset(next);
    const int L = first_scale(ctl->probe.emax, H);
    const int k1 = L / 2, k2 = L - L / 2;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ncomp;
         j += (int64_t)gridDim.x * blockDim.x) {
        const double v = (double)(long long)acc[j];
        src[j] = (v * __longlong_as_double((long long)(k1 + 1023) << 52)) *
                 __longlong_as_double((long long)(k2 + 1023) << 52);
    }
}

int quant_nbits(int64_t n_bound)
{
    int nb = 1;
    while (nb < 62 && ((int64_t)1 << nb) < n_bound) ++nb;
    return nb;
}

}  // namespace

extern "C" {

ST_API int64_t st_noalloc_max_cells(void) { return NOALLOC_MAX_CELLS; }

ST_API int st_step_noalloc(const st_params* p, const st_mesh_desc* m, int64_t n, double* x,
                           double* y, double* z, float* u, float* v, float* w, const float* d,
                           const float* U, double* source, double dt, double fluid_scale,
                           void* stream)
{
    if (!p || !m) return fail(ST_ERR_INVALID_ARGUMENT, "null params or mesh");
    if (p->precision != ST_PREC_MIXED || p->deposit != ST_DEPOSIT_DETERMINISTIC ||
        p->n_clouds != 1)
        return fail(ST_ERR_INVALID_ARGUMENT,
                    "st_step_noalloc supports mixed precision, the deterministic deposit and "
                    "one cloud");
    if (p->drag_model != ST_DRAG_STOKES_IMPLICIT && p->drag_model != ST_DRAG_SCHILLER_NAUMANN)
        return fail(ST_ERR_INVALID_ARGUMENT, "unknown drag model");
    if (p->n_substeps < 1) return fail(ST_ERR_INVALID_ARGUMENT, "n_substeps must be >= 1");
    if (!(p->mu_c > 0) || !(p->rho_c > 0) || !(p->rho_d > 0))
        return fail(ST_ERR_INVALID_ARGUMENT, "mu_c, rho_c and rho_d must be positive");
    if (!(dt > 0) || !(dt < 1e300)) return fail(ST_ERR_INVALID_ARGUMENT, "dt must be positive");
    int64_t ncells = 1;
    for (int a = 0; a < 3; ++a) {
        if (m->n[a] < 1 || !(m->ending[a] > m->origin[a]))
            return fail(ST_ERR_INVALID_ARGUMENT, "bad mesh");
        ncells *= m->n[a];
    }
    if (ncells > NOALLOC_MAX_CELLS)
        return fail(ST_ERR_INVALID_ARGUMENT,
                    "mesh too large for st_step_noalloc: at most st_noalloc_max_cells() "
                    "cells (the size of its fixed scratch array)");
    if (n < 0 || n > INT32_MAX) return fail(ST_ERR_INVALID_ARGUMENT, "parcel count out of range");
    if (n > 0 && (!x || !y || !z || !u || !v || !w || !d))
        return fail(ST_ERR_INVALID_ARGUMENT, "null parcel array");
    if (!U || !source) return fail(ST_ERR_INVALID_ARGUMENT, "null U or source");

    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES)
        return fail(ST_ERR_CUDA, "no current CUDA device");
    {
        /* the call synchronises the stream at its end, which a capture does not allow */
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        const cudaError_t e = cudaStreamIsCapturing(static_cast<cudaStream_t>(stream), &cs);
        if (e != cudaSuccess) return fail(ST_ERR_CUDA, cudaGetErrorString(e));
        if (cs != cudaStreamCaptureStatusNone)
            return fail(ST_ERR_INVALID_ARGUMENT,
                        "st_step_noalloc synchronises its stream and cannot be captured into a "
                        "CUDA graph");
    }
    Scratch sc;
    Turns::Turn turn;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        Scratch& g = g_scratch[dev];
        if (!g.acc) {
            void *pc = nullptr, *pa = nullptr;
            cudaError_t e = cudaGetSymbolAddress(&pc, g_st_noalloc_ctl);
            if (e == cudaSuccess) e = cudaGetSymbolAddress(&pa, g_st_noalloc_acc);
            if (e != cudaSuccess || !pc || !pa) return fail(ST_ERR_CUDA, cudaGetErrorString(e));
            int nsm = 148;
            cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
            for (int sub = 0; sub < 2; ++sub) {
                const int occ = step_max_active_blocks<double, float>(DEP_DET1, 256, sub + 1, 1);
                g.resident[sub] = nsm * (occ < 1 ? 1 : occ);
            }
            g.ctl = static_cast<CtlPair*>(pc);
            g.acc = static_cast<unsigned long long*>(pa);
        }
        sc = g;
        turn = g.turns.begin();
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Call call(dev, turn, s);
    CtlPair* const ctl = sc.ctl + turn.set;
    unsigned long long* const acc = sc.acc;
    const int64_t ncomp = ncells * 3;
    const int64_t resident = sc.resident[p->n_substeps > 1];

    const int64_t bound = n * (int64_t)p->n_substeps > 2 ? n * (int64_t)p->n_substeps : 2;
    const int H = 62 - QUANT_GROWTH_BITS - quant_nbits(bound);
    CloudK<double, float> ck;
    ck.x = x; ck.y = y; ck.z = z; ck.u = u; ck.v = v; ck.w = w; ck.d = d;
    ck.n = n;
    ck.tile0 = 0;
    ck.acc = acc;
    ck.src = nullptr;
    ck.cell = nullptr;

    StepArgs<double, float> a;
    for (int k = 0; k < 3; ++k) {
        a.mesh.N[k] = m->n[k];
        a.mesh.origin[k] = m->origin[k];
        a.mesh.rD[k] = 1.0 / ((m->ending[k] - m->origin[k]) / (double)m->n[k]);
    }
    a.mesh.NxNy = m->n[0] * m->n[1];
    a.mesh.pad = 0;
    a.mesh.nCells = ncells;
    a.phys.mu = (float)p->mu_c;
    a.phys.rho_d = (float)p->rho_d;
    a.phys.rr = (float)(p->rho_d / p->rho_c);
    a.phys.nu = (float)(p->mu_c / p->rho_c);
    a.phys.rnu = (float)(p->rho_c / p->mu_c);
    a.phys.alpha = (float)p->drag_multiplier;
    a.phys.dscale = (float)p->diameter_scale;
    a.phys.drag = p->drag_model;
    a.phys.nsub = p->n_substeps;
    a.dtP = dt / (double)p->n_substeps;
    a.dtV = (float)a.dtP;
    split_fluid_scale<double, float>(fluid_scale, a.fscale, a.fscale_lo);
    set_locate_bounds(a);
    a.nclouds = 1;
    a.U = U;
    a.clouds = nullptr;   /* one cloud: its descriptor is in the kernel parameters */
    a.ctl = &ctl->step;
    a.total_tiles = (n + WARP_TILE - 1) / WARP_TILE;
    a.one = ck;

    cudaError_t e;
    if (turn.reset) {
        k_noalloc_reset<<<1, 32, 0, s>>>(sc.ctl);
        if ((e = cudaGetLastError()) != cudaSuccess)
            return fail(ST_ERR_CUDA, cudaGetErrorString(e));
    }
    {
        /* with no parcels the probe still clears the accumulator */
        const int64_t need = (std::max(a.total_tiles, (ncomp + 31) / 32) + 7) / 8;
        StepArgs<double, float> probe = a;
        probe.ctl = &ctl->probe;
        probe.clear = acc;
        probe.clear_n = ncomp;
        e = launch_step<double, float>(probe, DEP_PROBE, (int)std::min(need, resident),
                                       256, s, false);
        if (e != cudaSuccess) return fail(ST_ERR_CUDA, cudaGetErrorString(e));
    }
    if (n > 0) {
        const int64_t need = (a.total_tiles + 7) / 8;
        a.probed = &ctl->probe;
        a.H = H;
        e = launch_step<double, float>(a, DEP_DET1, (int)std::min(need, resident), 256,
                                       s, true);
        if (e != cudaSuccess) return fail(ST_ERR_CUDA, cudaGetErrorString(e));
    }
    const int fgrid = (int)std::min<int64_t>((ncomp + 255) / 256, 148 * 8);
    e = launch_kernel(true, k_noalloc_finalize, dim3(fgrid), dim3(256), 0, s, acc, ctl,
                      sc.ctl + (turn.set ^ 1), H, source, ncomp);
    if (e != cudaSuccess) return fail(ST_ERR_CUDA, cudaGetErrorString(e));

    CloudCtl out;
    if ((e = cudaMemcpyAsync(&out, &ctl->step, sizeof out, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
        (e = cudaStreamSynchronize(s)) != cudaSuccess)
        return fail(ST_ERR_CUDA, cudaGetErrorString(e));
    call.complete = true;
    if (out.lost) return fail(ST_ERR_PARCEL_OUTSIDE, "parcel(s) could not be located in the mesh");
    if (out.overflow)
        return fail(ST_ERR_SOURCE_RANGE, "deposit(s) exceeded the fixed-point range");
    return ST_OK;
}

}  // extern "C"
