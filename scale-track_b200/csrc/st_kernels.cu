/*
 * st_kernels.cu -- the parcel step and the source reduction, written for sm_100a.
 *
 * One warp owns a tile of 32 consecutive parcels; lanes read the SoA arrays with
 * consecutive addresses (streaming loads, issued one tile ahead, that do not displace the
 * L2-resident cell arrays), gather the cell velocity, run the substeps in registers and
 * write back.
 * The deposit of each parcel into its cell (A:1342-1345, A:1361) is reduced inside the warp
 * over runs of equal cells (parcels are kept Morton-sorted by cell, so neighbours mostly
 * share a cell) and only the last lane of each run touches memory.
 *
 * Deterministic deposit: every deposit component is scaled by 2^-L and rounded to a 64-bit
 * integer, so the per-cell sums are integer sums and do not depend on which warp adds
 * first.  L follows the largest deposit of the previous step (CloudCtl).  With one limb the
 * headroom covers any distribution of the cloud's deposits over cells; two limbs (FP64
 * mode) carry 32 more bits of resolution.  A finalize pass converts the integers to FP64
 * and clears the accumulators for the next step.
 *
 * Reference: A: run/icoJuliaParcelFoam/cavity3D/asyncParallelTracking.jl
 *   evolve_on_device!  A:1258-1269     evolve_particle!  A:1271-1365
 *   locate             A:663-697       update! (GPU)     A:710-728
 * Compiled with --fmad=false: the reference's arithmetic has no fused multiply-adds.
 */
#include <cstdint>
#include <cuda_runtime.h>

#include "st_step.cuh"

namespace st {

/* ------------------------------------------------------------------------------------ */
/* the step kernel                                                                      */
/* ------------------------------------------------------------------------------------ */

constexpr int TILE = WARP_TILE;      /* parcels per warp tile (CloudK::tile0 counts these) */
constexpr int SLICES = TILE / 32;    /* 32-parcel slices per warp tile */

template <class P, class V>
__device__ __forceinline__ int find_cloud(const StepArgs<P, V>& a, int64_t tile)
{
    int lo = 0, hi = a.nclouds - 1;
    while (lo < hi) {  /* last cloud whose tile0 <= tile */
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(&a.clouds[mid].tile0) <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

/* The step kernel.  A warp owns a tile of SLICES x 32 consecutive parcels (lane l holds
 * parcels l, l+32, l+64, l+96 of the tile): all loads of the tile are issued one tile ahead
 * (while the previous tile is stepped), then the start cells are located and the cell
 * velocities gathered for every slice, then each slice is stepped, stored and its deposits
 * reduced.  Tiles are distributed over the persistent grid with a fixed stride; the clouds
 * of a multi-cloud launch occupy consecutive tile ranges. */
/* Resident blocks of 256 threads per SM the compiler must allow (a register budget):
 * 3 (80 registers), which holds the two tiles of the software pipeline without spills; FP64
 * velocities with one substep 2 (128 registers; 80 spill: 1e5 parcels 17.2 -> 15.0 us per
 * step, 4e5 26.6 -> 24.9 us).  Several substeps stay at 3 in every precision (mixed, 4e6
 * parcels with ten substeps: 2 blocks 373 us, 3 blocks 333 us, 4 blocks 430 us; FP64, 2e6 with
 * four: 2 blocks 180 us, 3 blocks 164 us). */
#ifndef ST_MIN_BLOCKS
#define ST_MIN_BLOCKS 3
#endif
#ifndef ST_MIN_BLOCKS_FP64
#define ST_MIN_BLOCKS_FP64 2
#endif
/* Several substeps per call (the multi-cloud workload) keep more state live per parcel. */
#ifndef ST_MIN_BLOCKS_SUB
#define ST_MIN_BLOCKS_SUB 3
#endif
template <class V, bool ONE>
struct MinBlocks {
    static constexpr int value =
        ONE ? (sizeof(V) == 8 ? ST_MIN_BLOCKS_FP64 : ST_MIN_BLOCKS) : ST_MIN_BLOCKS_SUB;
};

template <class P, class V, int DEP, bool ONE, bool SINGLE>
__global__ void __launch_bounds__(256, MinBlocks<V, ONE>::value) k_step(const StepArgs<P, V> a)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    constexpr bool DET = (DEP == DEP_DET1 || DEP == DEP_DET2);

    __shared__ __align__(16) unsigned long long dep_ws[8][dep_ws_words<DEP, V>];
    unsigned long long* const ws = dep_ws[threadIdx.x >> 5];
    grid_dep_launch();
    if (!ONE && sizeof(V) == 4 && a.phys.drag != 0) {   /* the table of x^0.687 serves the multi-substep loop */
        pow_tab_fill();
        __syncthreads();
    }
    grid_dep_wait();
    if (DEP == DEP_PROBE && a.clear) {
        for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < a.clear_n;
             j += (int64_t)gridDim.x * blockDim.x)
            a.clear[j] = 0ULL;
    }
    int cur = -1;
    /* in shared memory: nine registers less through the substeps */
    __shared__ Quant s_qp[8];
    Quant& qp = s_qp[threadIdx.x >> 5];
    AmaxT<V> amax = (V)0;
    unsigned ovf = 0, nlost = 0;

    /* Software pipeline over the warp's tiles (one substep): the streaming loads of the next
     * tile are issued before the current tile is stepped, so each warp keeps two tiles of
     * parcel data in flight and the HBM latency overlaps the arithmetic.  With several
     * substeps the kernel is bound by their arithmetic, the loads are a small share of it,
     * and the second tile's registers would spill in the substep loop: each tile is loaded
     * when it is stepped. */
    constexpr bool AHEAD = ONE;
    struct Raw {
        P X[SLICES], Y[SLICES], Z[SLICES];
        V Uv[SLICES], Vv[SLICES], Wv[SLICES], D[SLICES];
    };
    auto load = [&](int64_t t, Raw& r) {   /* every load of tile t (streaming, evict-first) */
        const int cc = SINGLE ? 0 : find_cloud(a, t);
        const CloudK<P, V>& cl = SINGLE ? a.one : a.clouds[cc];
        const int64_t n = cl.n;
        const int64_t base = (t - cl.tile0) * TILE + lane;
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
            const int64_t i = base + 32 * s;
            if (i < n) {
                r.X[s] = ld_stream(cl.x + i);
                r.Y[s] = ld_stream(cl.y + i);
                r.Z[s] = ld_stream(cl.z + i);
                r.Uv[s] = ld_stream(cl.u + i);
                r.Vv[s] = ld_stream(cl.v + i);
                r.Wv[s] = ld_stream(cl.w + i);
                r.D[s] = ld_stream(cl.d + i);
            }
        }
    };
    Raw R, RN;
    if (AHEAD && warp0 < a.total_tiles) load(warp0, R);
    for (int64_t tile = warp0; tile < a.total_tiles; tile += nwarps) {
        if (!AHEAD)
            load(tile, R);
        else if (tile + nwarps < a.total_tiles)
            load(tile + nwarps, RN);
        const int c = SINGLE ? 0 : find_cloud(a, tile);
        if (c != cur) {
            if (cur >= 0) flush_ctl<DEP>(a.ctl + cur, lane, amax, ovf, nlost);
            cur = c;
            if (DET) {
                const Quant q = SINGLE && a.probed
                                    ? make_quant(first_scale(a.probed->emax, a.H),
                                                 a.H + QUANT_GROWTH_BITS)
                                    : make_quant(a.ctl[c].L, a.ctl[c].H + QUANT_GROWTH_BITS);
                __syncwarp();
                if (lane == 0) qp = q;
                __syncwarp();
            }
        }
        const CloudK<P, V>& cl = SINGLE ? a.one : a.clouds[c];
        const int64_t n = cl.n;
        const int64_t base = (tile - cl.tile0) * TILE + lane;
        unsigned long long* const acc = DET ? cl.acc : nullptr;
        double* const src = (DEP == DEP_ATOMIC) ? cl.src : nullptr;
        P X[SLICES], Y[SLICES], Z[SLICES];
        V Uv[SLICES], Vv[SLICES], Wv[SLICES], D[SLICES];
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
            X[s] = R.X[s]; Y[s] = R.Y[s]; Z[s] = R.Z[s];
            Uv[s] = R.Uv[s]; Vv[s] = R.Vv[s]; Wv[s] = R.Wv[s]; D[s] = R.D[s];
        }
        if (AHEAD) R = RN;
        /* phase 2: start cells (A:1286) and raw cell velocities (A:1288; the fluid factor is
         * applied in the slip) */
        LocK st0[SLICES];
        V Ur[SLICES][3];
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
            st0[s].posI = 0;
            if (base + 32 * s < n) {
                bool bad = false;
                const LocK l0 = locate(a.mesh, X[s], Y[s], Z[s], bad);
                if (!bad && l0.part == 1) {
                    st0[s] = l0;
                    const V* Uc = a.U + 3 * (int64_t)(l0.posI - 1);
                    Ur[s][0] = __ldg(Uc);
                    Ur[s][1] = __ldg(Uc + 1);
                    Ur[s][2] = __ldg(Uc + 2);
                } else {
                    ++nlost;
                }
            }
        }
        /* phase 3: substeps, store, deposit, one slice after the other */
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
            const int64_t i = base + 32 * s;
            int32_t key = -1;
            V dep[3] = {(V)0, (V)0, (V)0};
            if (st0[s].posI > 0) {
                P pos[3] = {X[s], Y[s], Z[s]};
                V vel[3] = {Uv[s], Vv[s], Wv[s]};
                bool lost = false;
                if (ONE) {
                    evolve_one<P, V, false>(a, pos, vel, D[s] * a.phys.dscale, st0[s].posI,
                                     interior(a.mesh, st0[s]), Ur[s], lost, dep);
                    key = st0[s].posI - 1;
                } else {
                    evolve_parcel<P, V, DEP>(a, pos, vel, D[s] * a.phys.dscale, st0[s], Ur[s],
                                             acc, src, qp, amax, ovf, lost, key, dep);
                }
                if (lost) {
                    ++nlost;
                    key = -1;
                } else if (DEP != DEP_PROBE) {                                   /* A:1355-1360 */
                    /* the array pointers are read here, after the substeps, not held in
                     * registers through them */
                    st_stream(cl.x + i, pos[0]);
                    st_stream(cl.y + i, pos[1]);
                    st_stream(cl.z + i, pos[2]);
                    st_stream(cl.u + i, vel[0]);
                    st_stream(cl.v + i, vel[1]);
                    st_stream(cl.w + i, vel[2]);
                }
            }
            deposit_warp<DEP, V>(key, dep, acc, src, qp, lane, amax, ovf, ws);
        }
    }
    if (cur >= 0) flush_ctl<DEP>(a.ctl + cur, lane, amax, ovf, nlost);
}

template <class P, class V, bool ONE, bool SINGLE>
static cudaError_t launch_step_t(const StepArgs<P, V>& a, int dep, int grid, int block,
                                 cudaStream_t s, bool pdl)
{
    switch (dep) {
    case det_mode<V>: return launch_kernel(pdl, k_step<P, V, det_mode<V>, ONE, SINGLE>, grid, block, 0, s, a);
    case DEP_ATOMIC: return launch_kernel(pdl, k_step<P, V, DEP_ATOMIC, ONE, SINGLE>, grid, block, 0, s, a);
    case DEP_PROBE: return launch_kernel(pdl, k_step<P, V, DEP_PROBE, ONE, SINGLE>, grid, block, 0, s, a);
    default: return cudaErrorInvalidValue;
    }
}

template <class P, class V>
cudaError_t launch_step(const StepArgs<P, V>& a, int dep, int grid, int block, cudaStream_t s,
                        bool pdl)
{
    if (a.nclouds == 1)
        return a.phys.nsub == 1 ? launch_step_t<P, V, true, true>(a, dep, grid, block, s, pdl)
                                : launch_step_t<P, V, false, true>(a, dep, grid, block, s, pdl);
    return a.phys.nsub == 1 ? launch_step_t<P, V, true, false>(a, dep, grid, block, s, pdl)
                            : launch_step_t<P, V, false, false>(a, dep, grid, block, s, pdl);
}

template <class P, class V, bool ONE, bool SINGLE>
static int max_active_t(int dep, int block)
{
    int nb = 0;
    cudaError_t e = cudaErrorInvalidValue;
    switch (dep) {
    case det_mode<V>: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_step<P, V, det_mode<V>, ONE, SINGLE>, block, 0); break;
    case DEP_ATOMIC: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_step<P, V, DEP_ATOMIC, ONE, SINGLE>, block, 0); break;
    case DEP_PROBE: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_step<P, V, DEP_PROBE, ONE, SINGLE>, block, 0); break;
    default: break;
    }
    return e == cudaSuccess ? nb : 0;
}

/* Of the instance that runs: with FP64 velocities those of one substep are bounded at fewer
 * blocks than the others (MinBlocks).  With the smallest count over all instances the others
 * ran on two thirds of the grid (FP64, 2e6 parcels on 64^3 cells, four substeps: 188 against
 * 153 us per launch; 64 clouds, ten substeps: 2495 against 2181 us). */
template <class P, class V>
int step_max_active_blocks(int dep, int block, int nsub, int nclouds)
{
    if (nclouds == 1)
        return nsub == 1 ? max_active_t<P, V, true, true>(dep, block)
                         : max_active_t<P, V, false, true>(dep, block);
    return nsub == 1 ? max_active_t<P, V, true, false>(dep, block)
                     : max_active_t<P, V, false, false>(dep, block);
}

template cudaError_t launch_step<float, float>(const StepArgs<float, float>&, int, int, int, cudaStream_t,
                                                  bool);
template cudaError_t launch_step<double, float>(const StepArgs<double, float>&, int, int, int, cudaStream_t,
                                                  bool);
template cudaError_t launch_step<double, double>(const StepArgs<double, double>&, int, int, int, cudaStream_t,
                                                  bool);
template int step_max_active_blocks<float, float>(int, int, int, int);
template int step_max_active_blocks<double, float>(int, int, int, int);
template int step_max_active_blocks<double, double>(int, int, int, int);

/* ------------------------------------------------------------------------------------ */
/* source finalize: fixed point -> FP64, clear accumulators, next scale                 */
/* ------------------------------------------------------------------------------------ */

/* 32-byte accesses (one 32-byte sector per thread): two 16-byte accesses at a 32-byte stride
 * would touch every sector twice. */
__device__ __forceinline__ void ld32(const unsigned long long* p, unsigned long long v[4])
{
    asm volatile("ld.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
                 : "l"(__cvta_generic_to_global(p)));
}
__device__ __forceinline__ void st32(unsigned long long* p, unsigned long long v)
{
    asm volatile("st.global.v4.u64 [%0], {%1, %1, %1, %1};" ::"l"(__cvta_generic_to_global(p)),
                 "l"(v)
                 : "memory");
}
__device__ __forceinline__ void st32_stream(double* p, const double v[4])
{
    asm volatile("st.global.cs.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(
                     __cvta_generic_to_global(p)),
                 "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3])
                 : "memory");
}

/* What bounds it is traffic: the accumulator read, the source written, the accumulator cleared
 * for the step after.  CLEAR: the clearing here, of the groups of four components that hold
 * something (few with small clouds on a shared mesh: 64 sources of 64^3 cells, 403 MB each of
 * accumulators and sources, 207 us; 171 us and a memset of 75 us without).  The source is
 * written whole, zeros included: callers hold its device pointer. */
template <int LIMBS, bool CLEAR>
__global__ void __launch_bounds__(256) k_finalize(unsigned long long* __restrict__ acc,
                                                  double* __restrict__ src,
                                                  float* __restrict__ src32, CloudCtl* ctl,
                                                  const int32_t* Lsrc,
                                                  unsigned int* counter, int nclouds,
                                                  int64_t stride)
{
    grid_dep_launch();
    grid_dep_wait();
    /* stride: per-cloud component count, a multiple of 4 (padding stays zero).  Lsrc: the
     * scale of each cloud when the next scale was already set by k_next_scale (overlapped
     * finalize), else null. */
    const int c = blockIdx.y;
    const int L = Lsrc ? Lsrc[c] : ctl[c].L;
    unsigned long long* const a = acc + (int64_t)c * stride * LIMBS;
    double* const s = src + (int64_t)c * stride;
    float4* const s32 = src32 ? reinterpret_cast<float4*>(src32 + (int64_t)c * stride) : nullptr;
    const int64_t ngroups = stride / 4;
    const int64_t gstride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < ngroups; g += gstride) {
        unsigned long long q[4 * LIMBS];
        unsigned long long any = 0;
#pragma unroll
        for (int l = 0; l < LIMBS; ++l) {
            const unsigned long long* const p = a + 4 * (LIMBS * g + l);
            if (CLEAR) {
                ld32(p, q + 4 * l);
            } else {
                const ulonglong2 q0 = __ldcs(reinterpret_cast<const ulonglong2*>(p));
                const ulonglong2 q1 = __ldcs(reinterpret_cast<const ulonglong2*>(p) + 1);
                q[4 * l] = q0.x;
                q[4 * l + 1] = q0.y;
                q[4 * l + 2] = q1.x;
                q[4 * l + 3] = q1.y;
            }
        }
#pragma unroll
        for (int k = 0; k < 4 * LIMBS; ++k) any |= q[k];
        double o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            double v;
            if (LIMBS == 1) {
                v = (double)(long long)q[k];
            } else {
                long long hi = (long long)q[2 * k];
                unsigned long long lo = q[2 * k + 1];
                hi += (long long)(lo >> 32);
                lo &= 0xffffffffULL;
                v = (double)hi * 4294967296.0 + (double)lo;
            }
            o[k] = ldexp2(v, L);
        }
        if (CLEAR) {
            st32_stream(s + 4 * g, o);
        } else {
            __stcs(reinterpret_cast<double2*>(s + 4 * g), make_double2(o[0], o[1]));
            __stcs(reinterpret_cast<double2*>(s + 4 * g) + 1, make_double2(o[2], o[3]));
        }
        if (CLEAR && any) {
#pragma unroll
            for (int l = 0; l < LIMBS; ++l) st32(a + 4 * (LIMBS * g + l), 0ULL);
        }
        /* a 4-byte copy for an FP32 exchange array, rounded once from the FP64 source */
        if (s32) __stcs(s32 + g, make_float4((float)o[0], (float)o[1], (float)o[2], (float)o[3]));
    }
    /* the last block to finish moves every cloud to the scale of its largest deposit */
    if (Lsrc) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        unsigned int ticket = atomicAdd(counter, 1u);
        if (ticket == gridDim.x * gridDim.y - 1) {
            __threadfence();
            for (int k = 0; k < nclouds; ++k) {
                volatile CloudCtl* q = ctl + k;
                int em = q->emax;
                if (em != EXP_NONE) q->L = em - q->H;
                q->emax = EXP_NONE;
            }
            *counter = 0u;
            __threadfence();
        }
    }
}

/* Where the accumulators are cleared.  Those of one cloud, small ones, and those far larger than
 * the L2, by the conversion (15 MB of accumulators, three handles in turn: 35 against 39 us per
 * pass of two steps; 403 MB: 1207 against 1386 us; one cloud on 1.6e6 tets, 38 MB: 62.6 against
 * 66 us).  Between, where the accumulators of many clouds fit the L2 but not along with all
 * else, they are read evict-first and a memset of its own leaves their zeros in the L2 for the
 * step's adds (three handles in turn, by the memset and by the conversion: 33 MB 145 and 165 us;
 * 36 MB 84 and 90; 84 MB 217 and 220).  One handle alone is faster with the conversion there too
 * (64^3 cells, two steps: 31 MB 75.5 and 53.9 us, 82 MB 150 and 125; 50 MB in FP64 88.9 and 63.4):
 * the lines are drawn for programs with several handles.  Outside them both agree on the
 * conversion (19 MB 60.2 and 47.6 us; 126 MB 217 and 204). */
cudaError_t launch_finalize(int limbs, unsigned long long* acc, double* src, float* src32,
                            CloudCtl* ctl, const int32_t* Lsrc, unsigned int* counter,
                            int nclouds, int64_t stride, int grid_x, cudaStream_t s, bool pdl)
{
    if (stride % 4) return cudaErrorInvalidValue;
    const size_t bytes = (size_t)stride * nclouds * limbs * 8;
    const bool clear = nclouds == 1 || bytes <= (size_t)24 << 20 || bytes > (size_t)96 << 20;
    const auto k = limbs == 1 ? (clear ? k_finalize<1, true> : k_finalize<1, false>)
                              : (clear ? k_finalize<2, true> : k_finalize<2, false>);
    const cudaError_t e = launch_kernel(pdl && clear, k, dim3(grid_x, nclouds), dim3(256), 0, s,
                                        acc, src, src32, ctl, Lsrc, counter, nclouds, stride);
    if (e != cudaSuccess || clear) return e;
    return cudaMemsetAsync(acc, 0, bytes, s);
}

/* The scale bookkeeping of k_finalize on its own, for an overlapped finalize: keeps each
 * cloud's scale of the step just run in Lfin (for the finalize on the other stream) and moves
 * the cloud to the scale of that step's largest deposit for the next step. */
__global__ void k_next_scale(CloudCtl* ctl, int32_t* Lfin, int nclouds)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nclouds) {
        Lfin[k] = ctl[k].L;
        const int em = ctl[k].emax;
        if (em != EXP_NONE) ctl[k].L = em - ctl[k].H;
        ctl[k].emax = EXP_NONE;
    }
}

cudaError_t launch_next_scale(CloudCtl* ctl, int32_t* Lfin, int nclouds, cudaStream_t s)
{
    k_next_scale<<<(nclouds + 127) / 128, 128, 0, s>>>(ctl, Lfin, nclouds);
    return cudaGetLastError();
}

/* After a probe pass: the scale of the first step maps the largest deposit to 2^H. */
__global__ void k_set_scale(CloudCtl* ctl, int nclouds)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nclouds) {
        int em = ctl[k].emax;
        ctl[k].L = first_scale(em, ctl[k].H);
        ctl[k].emax = EXP_NONE;
    }
}

/* Copies every cloud's largest-deposit exponent between the control blocks and a contiguous
 * array (to_ctl: array -> blocks), the buffer a sharded run max-reduces across ranks. */
__global__ void k_ctl_exponents(CloudCtl* ctl, int32_t* e, int nclouds, int to_ctl)
{
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nclouds) {
        if (to_ctl) ctl[k].emax = e[k];
        else e[k] = ctl[k].emax;
    }
}

cudaError_t launch_ctl_exponents(CloudCtl* ctl, int32_t* e, int nclouds, bool to_ctl,
                                 cudaStream_t s)
{
    k_ctl_exponents<<<(nclouds + 127) / 128, 128, 0, s>>>(ctl, e, nclouds, to_ctl ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_set_scale(CloudCtl* ctl, int nclouds, cudaStream_t s)
{
    k_set_scale<<<(nclouds + 127) / 128, 128, 0, s>>>(ctl, nclouds);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(256) k_zero_f64(double* p, int64_t n)
{
    grid_dep_launch();
    grid_dep_wait();
    /* n is a multiple of 4 and p 32-byte aligned (padded per-cloud strides) */
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n / 4;
         j += (int64_t)gridDim.x * blockDim.x)
        st32(reinterpret_cast<unsigned long long*>(p) + 4 * j, 0ULL);
}

cudaError_t launch_zero_f64(double* p, int64_t n, cudaStream_t s, bool pdl)
{
    const int64_t g = (n / 4 + 255) / 256;
    const int grid = (int)(g < 1 ? 1 : (g < 148 * 8 ? g : 148 * 8));
    return launch_kernel(pdl, k_zero_f64, dim3(grid), dim3(256), 0, s, p, n);
}

__global__ void k_f64_to_f32(const double* __restrict__ in, float* __restrict__ out, int64_t n)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x)
        out[j] = (float)in[j];
}

/* Element-wise conversion between FP32 and FP64 arrays; either side may be mapped host
 * memory (the zero-copy exchange reads U from and writes the source to it directly). */
template <class I, class O>
__global__ void k_convert(const I* __restrict__ in, O* __restrict__ out, int64_t n)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x)
        out[j] = (O)in[j];
}

cudaError_t launch_convert(const void* in, int in_bytes, void* out, int out_bytes, int64_t n,
                           cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    int64_t g = (n + 255) / 256;
    if (g > 148 * 16) g = 148 * 16;
    if (in_bytes == 4 && out_bytes == 4)
        k_convert<float, float><<<(int)g, 256, 0, s>>>((const float*)in, (float*)out, n);
    else if (in_bytes == 4)
        k_convert<float, double><<<(int)g, 256, 0, s>>>((const float*)in, (double*)out, n);
    else if (out_bytes == 4)
        k_convert<double, float><<<(int)g, 256, 0, s>>>((const double*)in, (float*)out, n);
    else
        k_convert<double, double><<<(int)g, 256, 0, s>>>((const double*)in, (double*)out, n);
    return cudaGetLastError();
}

/* Constant extrapolation of the source (A:742-747): est = 2 S - est_prev, in place on
 * `est`, with S = 0 when there is no completed step yet (s == nullptr); the FP32 copy for a
 * 4-byte exchange array is written alongside. */
__global__ void k_extrapolate(const double* __restrict__ s, double* __restrict__ est,
                             float* __restrict__ est32, int64_t n)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x) {
        const double e = (s ? 2.0 * s[j] : 0.0) - est[j];
        est[j] = e;
        if (est32) est32[j] = (float)e;
    }
}

cudaError_t launch_extrapolate(const double* s, double* est, float* est32, int64_t n,
                               cudaStream_t st)
{
    int64_t g = (n + 255) / 256;
    if (g > 148 * 8) g = 148 * 8;
    if (g < 1) g = 1;
    k_extrapolate<<<(int)g, 256, 0, st>>>(s, est, est32, n);
    return cudaGetLastError();
}

__global__ void k_f32_to_f64(const float* __restrict__ in, double* __restrict__ out, int64_t n)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
         j += (int64_t)gridDim.x * blockDim.x)
        out[j] = (double)in[j];
}

cudaError_t launch_f64_to_f32(const double* in, float* out, int64_t n, cudaStream_t s)
{
    int grid = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
    if (grid < 1) grid = 1;
    k_f64_to_f32<<<grid, 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}

cudaError_t launch_f32_to_f64(const float* in, double* out, int64_t n, cudaStream_t s)
{
    int grid = (int)((n + 255) / 256 < 148 * 8 ? (n + 255) / 256 : 148 * 8);
    if (grid < 1) grid = 1;
    k_f32_to_f64<<<grid, 256, 0, s>>>(in, out, n);
    return cudaGetLastError();
}

}  // namespace st
