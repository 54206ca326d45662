/*
 * st_adjoint.cu -- adjoint of the parcel step for the time-averaged source (no counterpart
 * in the reference, which has no adjoint).
 *
 * Objective-side contract (the pull-back of y = Sbar = (1/T) sum_n S_n): given the cotangent
 * ybar = dJ/dSbar per cell, return dJ/dalpha (drag multiplier), dJ/ds (diameter scale) and
 * dJ/dv0 per parcel, with cell ownership and wall-bounce decisions frozen at the forward
 * pass.  Schiller-Naumann drag, one substep.  Mathematics (forward and reverse step):
 *   u = U[c_n] fs_n, d_e = s d, f = 18 mu dt alpha / (rho_d d_e^2), du = u - v,
 *   Re = |du| d_e rnu, P = Re^0.687, g = f (1 + 0.15 P)
 *   v'_k = v_k + g du_k  (-v_k if bounced),  D_k = m (v_k - v'_k)  (0 if bounced)
 *   w_k = a_k - m G_k (not bounced), Sw = sum w_k du_k, gamma = 0.10305 f P / |du|^2
 *   a_j <- [not bounced]((1-g) w_j + m G_j) - [bounced] a_j - gamma du_j Sw
 *   dJ/dalpha += Sw g / alpha,  dJ/ds += Sw (-2g + 0.10305 f P)/s + (3/s) sum G_k D_k
 * with G = ybar / T.
 *
 * Kernels: k_adj_forward runs all T steps of a parcel in registers (the mean-source
 * objective only needs the sum over steps), writes checkpoints of (x, v) every C steps and
 * deposits every step into one fixed-point accumulator with a constant scale, a parcel's
 * deposits into one cell summed in registers first.  k_adj_reverse takes 256 parcels per block at a time from
 * the last checkpoint segment to the first: it recomputes the C forward steps of a segment,
 * recording what the reverse step needs, then runs the reverse steps back to the checkpoint,
 * keeping the parcels' cotangents and FP64 parameter partials in registers through all
 * segments.  Parameter partials are reduced per 256 parcels in shared memory in a fixed order
 * and summed on the host in parcel order, so the gradient is reproducible.
 *
 * What bounds them: instruction issue (the step's arithmetic, 200 steps per parcel for one
 * load).  What depends on the parcel alone is formed once, and the cell located at the end of
 * a step is the start cell of the next unless the parcel bounced.  The records are held per
 * resident block, not per parcel, so that they stay in the L2 between writing and reading.
 * 1e6 parcels on 128^3 cells, 200 steps, checkpoints every 20, mixed precision: forward
 * 3.89 -> 1.75 ms (2.96 ms with every step's deposits going to memory), reverse 3.88 -> 2.63 ms
 * (records per parcel in HBM, power and cell velocity formed again in the reverse step before).
 */
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "st_step.cuh"

namespace st {

/* What a step of one parcel keeps from its diameter: m/rho_c and the drag factor. */
template <class V>
struct AdjParcel {
    V mB, f;
};

template <class P, class V>
__device__ __forceinline__ AdjParcel<V> adj_parcel(const AdjArgs<P, V>& a, V d)
{
    const PhysK<V>& ph = a.phys;
    AdjParcel<V> r;
    r.mB = ((ph.rr * (V)3.14159265358979323846) * ((d * d) * d)) / (V)6;
    r.f = ((((V)18 * ph.mu) * a.dtV) / (ph.rho_d * (d * d))) * ph.alpha;
    return r;
}

/* Start cell of the next step: posI is 1-based, ok = located inside the mesh. */
struct AdjCell {
    int32_t posI;
    bool ok;
};

template <class P>
__device__ __forceinline__ AdjCell adj_cell(const MeshK<P>& m, const P x[3])
{
    bool bad = false;
    const LocK l = locate(m, x[0], x[1], x[2], bad);
    return {l.posI, !bad && l.part == 1};
}

template <class V>
struct AdjLocal {
    V du[3];   /* slip velocity */
    V pw;      /* Re^0.687 */
    V dep[3];  /* the step's deposit */
};

template <class V>
__device__ __forceinline__ V adj_pow(V Re)
{
    if (sizeof(V) == 4) return (V)pow0687f((float)Re);
    return (V)st_pow0687((double)Re);
}

/* One forward step (evolve_particle!, nSteps = 1) from start cell c, which becomes that of
 * the next step; b = bounce flags.  Returns false if the parcel is lost. */
template <class P, class V>
__device__ __forceinline__ bool adj_step(const AdjArgs<P, V>& a, const AdjParcel<V>& q, P pos[3],
                                         V vel[3], V d, V fs, V fs_lo, AdjCell& c, unsigned& b,
                                         AdjLocal<V>& o)
{
    constexpr bool MIX = is_mixed<P, V>;
    const MeshK<P>& m = a.mesh;
    b = 0;
    if (!c.ok) return false;
    const int32_t posI = c.posI;
    const V* Uc = a.U + 3 * (int64_t)(posI - 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) o.du[k] = slip<MIX>(__ldg(Uc + k), fs, fs_lo, vel[k]);
    const V mag = st_sqrt((o.du[0] * o.du[0] + o.du[1] * o.du[1]) + o.du[2] * o.du[2]);
    o.pw = adj_pow<V>((mag * d) * a.phys.rnu);
    const V g = q.f * ((V)1 + (V)0.15 * o.pw);
    P posNew[3];
    V velNew[3], inc[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        inc[k] = g * o.du[k];
        velNew[k] = vel[k] + inc[k];
        posNew[k] = pos[k] + (P)velNew[k] * a.dtP;
    }
    bool bad = false;
    const LocK ln = locate(m, posNew[0], posNew[1], posNew[2], bad);
    if (bad) return false;
    if (ln.posI != posI || ln.part != 1) {
        b = (ln.I < 0 || ln.I >= m.N[0] ? 1u : 0u) | (ln.J < 0 || ln.J >= m.N[1] ? 2u : 0u) |
            (ln.K < 0 || ln.K >= m.N[2] ? 4u : 0u);
    }
    c.posI = ln.posI;
    c.ok = ln.part == 1;
    V state0[3] = {vel[0], vel[1], vel[2]};
    if (b) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (b & (1u << k)) {
                posNew[k] = pos[k];
                velNew[k] = -vel[k];
                state0[k] -= (V)2 * vel[k];
            }
        }
        c = adj_cell(m, posNew);
    }
    /* deposit forms of the step kernel (st_step.cuh evolve_one): mixed precision deposits
     * -m/rho_c times the velocity increment, zero on a bounced component */
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if constexpr (MIX) o.dep[k] = q.mB * ((b & (1u << k)) ? (V)0 : -inc[k]);
        else o.dep[k] = q.mB * (state0[k] - velNew[k]);
        pos[k] = posNew[k];
        vel[k] = velNew[k];
    }
    return true;
}

/* What the reverse of a step needs of its forward: in mixed precision the slip velocity, in
 * FP64 the velocity at the start of the step (its deposit is the difference of two rounded
 * velocities), and Re^0.687. */
template <class V>
struct alignas(4 * sizeof(V)) AdjRec {
    V x[3];
    V pw;
};

/* Reverse step: av = cotangent after the step (in) and before it (out). */
template <class P, class V>
__device__ __forceinline__ void adj_reverse(const AdjArgs<P, V>& a, const AdjParcel<V>& q,
                                            const AdjRec<V>& r, V fs, V fs_lo, int32_t cell,
                                            unsigned b, V av[3], double& dalpha, double& dscale)
{
    constexpr bool MIX = is_mixed<P, V>;
    const PhysK<V>& ph = a.phys;
    const V* Gd = a.G + 3 * (int64_t)cell;
    const V G[3] = {__ldg(Gd), __ldg(Gd + 1), __ldg(Gd + 2)};
    V du[3];
    if constexpr (MIX) {
#pragma unroll
        for (int k = 0; k < 3; ++k) du[k] = r.x[k];
    } else {
        const V* Uc = a.U + 3 * (int64_t)cell;
#pragma unroll
        for (int k = 0; k < 3; ++k) du[k] = slip<MIX>(__ldg(Uc + k), fs, fs_lo, r.x[k]);
    }
    const V mag2 = (du[0] * du[0] + du[1] * du[1]) + du[2] * du[2];
    const V g = q.f * ((V)1 + (V)0.15 * r.pw);
    V dep[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const V inc = g * du[k];
        const bool bk = b & (1u << k);
        if constexpr (MIX) {
            dep[k] = q.mB * (bk ? (V)0 : -inc);
        } else {
            const V velNew = bk ? -r.x[k] : r.x[k] + inc;
            const V state0 = bk ? r.x[k] - (V)2 * r.x[k] : r.x[k];
            dep[k] = q.mB * (state0 - velNew);
        }
    }
    V w[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) w[k] = (b & (1u << k)) ? (V)0 : av[k] - q.mB * G[k];
    const V Sw = (w[0] * du[0] + w[1] * du[1]) + w[2] * du[2];
    const V gamma = mag2 > (V)0 ? (((V)0.10305 * q.f) * r.pw) / mag2 : (V)0;
    V an[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        const V t = (b & (1u << j)) ? -av[j] : ((V)1 - g) * w[j] + q.mB * G[j];
        an[j] = t - (gamma * du[j]) * Sw;
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) av[j] = an[j];
    /* division by one is exact: skipped (uniformly) for the common parameters */
    dalpha += (double)(Sw * (ph.alpha == (V)1 ? g : g / ph.alpha));
    const V GD = (G[0] * dep[0] + G[1] * dep[1]) + G[2] * dep[2];
    const V sw = Sw * ((V)-2 * g + ((V)0.10305 * q.f) * r.pw);
    dscale += (double)(ph.dscale == (V)1 ? sw + (V)3 * GD
                                         : sw / ph.dscale + ((V)3 / ph.dscale) * GD);
}

/* The fixed-point sum of a parcel's deposits since it entered its cell: only their sum over
 * the steps is wanted, so they go to memory when the parcel leaves the cell (one limb: q; two:
 * the high words in q, the low ones in lo).  The headroom bounds the sum of all deposits. */
template <class V>
struct AdjRun {
    int32_t key = -1;
    long long q[3] = {0, 0, 0};
    unsigned long long lo[3] = {0, 0, 0};

    __device__ __forceinline__ void flush(unsigned long long* acc)
    {
        if (key < 0) return;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if constexpr (sizeof(V) == 4) {
                if (q[k]) red_add(acc + 3 * (int64_t)key + k, (unsigned long long)q[k]);
            } else {
                if (q[k]) red_add(acc + 2 * (3 * (int64_t)key + k), (unsigned long long)q[k]);
                if (lo[k]) red_add(acc + 2 * (3 * (int64_t)key + k) + 1, lo[k]);
                lo[k] = 0;
            }
            q[k] = 0;
        }
    }
    __device__ __forceinline__ void add(const long long v[3])
    {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if constexpr (sizeof(V) == 4) {
                q[k] += v[k];
            } else {
                q[k] += v[k] >> 32;
                lo[k] += (unsigned long long)v[k] & 0xffffffffULL;
            }
        }
    }
};

/* MODE 0: probe (first step, largest |deposit| only).  MODE 1: all T steps with
 * checkpoints and the fixed-point mean-source accumulation. */
template <class P, class V, int MODE>
__global__ void __launch_bounds__(256) k_adj_forward(const AdjArgs<P, V> a)
{
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool active = i < a.n;
    P pos[3] = {(P)0, (P)0, (P)0};
    V vel[3] = {(V)0, (V)0, (V)0}, d = (V)1;
    if (active) {
        pos[0] = a.x[i]; pos[1] = a.y[i]; pos[2] = a.z[i];
        vel[0] = a.u[i]; vel[1] = a.v[i]; vel[2] = a.w[i];
        d = a.d[i] * a.phys.dscale;
    }
    const AdjParcel<V> q = adj_parcel(a, d);
    AdjCell c = {0, false};
    if (active) c = adj_cell(a.mesh, pos);
    bool alive = active;
    AmaxT<V> amax = (V)0;
    unsigned lost = 0, ovf = 0;
    const int nsteps = MODE == 0 ? 1 : a.T;
    /* fixed-point parameters of the mean accumulator (constant over the run) */
    Quant qp = {0.0, 0.0, 0.0f, 0.0f, 0, false};
    if (MODE == 1) qp = make_quant(a.ctl->L, a.ctl->H + QUANT_GROWTH_BITS);
    AdjRun<V> run;
    int until = 0;   /* steps until the next checkpoint */
    int64_t ck = 0;
    for (int n = 0; n < nsteps; ++n) {
        if (MODE == 1 && until-- == 0) {
            until = a.C - 1;
            if (active) {
                P* cx = a.ck_x + ck * 3 * a.n;
                V* cv = a.ck_v + ck * 3 * a.n;
                cx[i] = pos[0]; cx[a.n + i] = pos[1]; cx[2 * a.n + i] = pos[2];
                cv[i] = vel[0]; cv[a.n + i] = vel[1]; cv[2 * a.n + i] = vel[2];
            }
            ++ck;
        }
        if (!alive) continue;
        const int32_t cell = c.posI - 1;
        unsigned b;
        AdjLocal<V> o;
        if (!adj_step<P, V>(a, q, pos, vel, d, a.fs[n], a.fs_lo[n], c, b, o)) {
            alive = false;
            ++lost;
        } else if (MODE == 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) track_max(o.dep[k], amax);
        } else {
            if (cell != run.key) {
                run.flush(a.acc);
                run.key = cell;
            }
            long long v[3];
            quantize3(o.dep, qp, amax, ovf, v);
            run.add(v);
        }
    }
    if (MODE == 1) run.flush(a.acc);
    if (MODE == 0) {
        const int e = amax > (V)0 ? exp_of((double)amax) : EXP_NONE;
        const int wmax = __reduce_max_sync(FULL_MASK, e);
        if (lane == 0 && wmax != EXP_NONE) atomicMax(&a.ctl->emax, wmax);
    }
    const unsigned nl = __reduce_add_sync(FULL_MASK, lost);
    const unsigned no = __reduce_add_sync(FULL_MASK, ovf);
    if (lane == 0) {
        if (nl) atomicAdd(&a.ctl->lost, (unsigned long long)nl);
        if (no) atomicAdd(&a.ctl->overflow, (unsigned long long)no);
    }
}

/* The pull-back of 256 parcels at a time, all checkpoint segments from the last to the
 * first.  Records of a block, W = a.width: AdjRec[C][W], then cells int32[C][W] (-1: lost,
 * below that -2 - cell: bounced, flags in the bytes that follow), then flags uint8[C][W].
 * WIDE: the width is 256 as a constant; read from the arguments, in 64 bits, it takes 1 to 3 %
 * longer (300000 FP64 parcels, 200 steps: 1.584 -> 1.636 ms). */
/* Resident blocks: 3 (80 registers) in mixed precision, 4 in FP64 (3e5 parcels, 200 steps:
 * 1.83 ms with 3, 1.72 ms with 4). */
template <class P, class V, bool WIDE>
__global__ void __launch_bounds__(256, sizeof(V) == 8 ? 4 : 3) k_adj_reverse(const AdjArgs<P, V> a)
{
    __shared__ double red[2][256];
    const int tid = threadIdx.x;
    const std::conditional_t<WIDE, int, int64_t> W = WIDE ? 256 : a.width;
    unsigned char* const slot = a.rec + (int64_t)blockIdx.x * a.C * W * adj_rec_bytes<V>;
    AdjRec<V>* const rec = reinterpret_cast<AdjRec<V>*>(slot) + tid;
    int32_t* const rec_c =
        reinterpret_cast<int32_t*>(slot + (int64_t)a.C * W * sizeof(AdjRec<V>)) + tid;
    uint8_t* const rec_b =
        slot + (int64_t)a.C * W * (sizeof(AdjRec<V>) + sizeof(int32_t)) + tid;
    const int nseg = (a.T + a.C - 1) / a.C;
    const int64_t chunks = (a.n + 255) / 256;
    for (int64_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
        const int64_t i = ch * 256 + tid;
        double dalpha = 0.0, dscale = 0.0;
        if (i < a.n) {
            const V d = a.d[i] * a.phys.dscale;
            const AdjParcel<V> q = adj_parcel(a, d);
            V av[3] = {(V)0, (V)0, (V)0};
            for (int seg = nseg - 1; seg >= 0; --seg) {
                const P* cx = a.ck_x + (int64_t)seg * 3 * a.n;
                const V* cv = a.ck_v + (int64_t)seg * 3 * a.n;
                P pos[3] = {cx[i], cx[a.n + i], cx[2 * a.n + i]};
                V vel[3] = {cv[i], cv[a.n + i], cv[2 * a.n + i]};
                const int n0 = seg * a.C;
                const int len = min(a.C, a.T - n0);
                AdjCell c = adj_cell(a.mesh, pos);
                bool ok = true;
                for (int t = 0; t < len; ++t) {       /* recompute, recording the forward */
                    AdjRec<V> r = {{vel[0], vel[1], vel[2]}, (V)0};
                    const int32_t cell = c.posI - 1;
                    unsigned b = 0;
                    AdjLocal<V> o;
                    ok = ok && adj_step<P, V>(a, q, pos, vel, d, a.fs[n0 + t], a.fs_lo[n0 + t], c,
                                              b, o);
                    if (ok) {
                        r.pw = o.pw;
                        if constexpr (is_mixed<P, V>) {
#pragma unroll
                            for (int k = 0; k < 3; ++k) r.x[k] = o.du[k];
                        }
                        rec[t * W] = r;
                        if (b) rec_b[t * W] = (uint8_t)b;
                    }
                    rec_c[t * W] = !ok ? -1 : (b ? -2 - cell : cell);
                }
                int32_t cn = rec_c[(len - 1) * W];
                AdjRec<V> rn = rec[(len - 1) * W];
                for (int t = len - 1; t >= 0; --t) {  /* reverse, the next record in flight */
                    const int32_t cc = cn;
                    const AdjRec<V> r = rn;
                    if (t > 0) {
                        cn = rec_c[(t - 1) * W];
                        rn = rec[(t - 1) * W];
                    }
                    if (cc == -1) continue;
                    const unsigned b = cc < 0 ? rec_b[t * W] : 0u;
                    adj_reverse<P, V>(a, q, r, a.fs[n0 + t], a.fs_lo[n0 + t],
                                      cc < 0 ? -2 - cc : cc, b, av, dalpha, dscale);
                }
            }
            if (a.dv0) {                              /* in the order of st_set_parcels */
                const int64_t p = a.id[i];
#pragma unroll
                for (int k = 0; k < 3; ++k) a.dv0[k * a.n + p] = (double)av[k];
            }
        }
        red[0][tid] = dalpha;
        red[1][tid] = dscale;
        __syncthreads();
        for (int s = 128; s > 0; s >>= 1) {
            if (tid < s) {
                red[0][tid] += red[0][tid + s];
                red[1][tid] += red[1][tid + s];
            }
            __syncthreads();
        }
        if (tid < 2) a.partials[2 * ch + tid] = red[tid][0];
        __syncthreads();
    }
}

/* The cotangent of one step: G = ybar / T in FP64, rounded to the velocity type. */
template <class V>
__global__ void k_adj_cotangent(const double* __restrict__ ybar, double T, V* __restrict__ G,
                                int64_t ncomp)
{
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ncomp;
         j += (int64_t)gridDim.x * blockDim.x)
        G[j] = (V)(ybar[j] / T);
}

/* Mean source (1/T) * fixed point -> FP64, into `mean` [ncomp]. */
__global__ void k_adj_mean(const unsigned long long* __restrict__ acc, const CloudCtl* ctl,
                           int limbs, double T, double* __restrict__ mean, int64_t ncomp)
{
    const int L = ctl->L;
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < ncomp;
         j += (int64_t)gridDim.x * blockDim.x) {
        double v;
        if (limbs == 1) {
            v = (double)(long long)acc[j];
        } else {
            long long hi = (long long)acc[2 * j];
            unsigned long long lo = acc[2 * j + 1];
            hi += (long long)(lo >> 32);
            lo &= 0xffffffffULL;
            v = (double)hi * 4294967296.0 + (double)lo;
        }
        const int k1 = L / 2, k2 = L - L / 2;
        mean[j] = ((v * st_pow2i(k1)) * st_pow2i(k2)) / T;
    }
}

/* After the probe: a constant scale for the whole run. */
__global__ void k_adj_scale(CloudCtl* ctl)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        const int em = ctl->emax;
        ctl->L = (em == EXP_NONE) ? -ctl->H : em - ctl->H;
        ctl->emax = EXP_NONE;
    }
}

template <class P, class V>
cudaError_t launch_adj_forward(const AdjArgs<P, V>& a, bool probe, cudaStream_t s)
{
    const int grid = (int)((a.n + 255) / 256);
    if (grid == 0) return cudaSuccess;
    if (probe) k_adj_forward<P, V, 0><<<grid, 256, 0, s>>>(a);
    else k_adj_forward<P, V, 1><<<grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

template <class P, class V>
cudaError_t launch_adj_reverse(const AdjArgs<P, V>& a, int grid, cudaStream_t s)
{
    if (grid == 0) return cudaSuccess;
    /* the record indices of a block are below 256 * C */
    if (a.width == 256 && a.C < INT32_MAX / 256) k_adj_reverse<P, V, true><<<grid, 256, 0, s>>>(a);
    else k_adj_reverse<P, V, false><<<grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

/* Blocks of the reverse kernel: as many as stay resident, at most one per 256 parcels. */
template <class P, class V>
int adj_reverse_grid(int64_t n, int nsm)
{
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_adj_reverse<P, V, true>, 256, 0) !=
            cudaSuccess || nb < 1)
        nb = 1;
    const int64_t chunks = (n + 255) / 256;
    return (int)(chunks < (int64_t)nsm * nb ? chunks : (int64_t)nsm * nb);
}

template <class V>
cudaError_t launch_adj_cotangent(const double* ybar, int T, V* G, int64_t ncomp, cudaStream_t s)
{
    const int64_t g = (ncomp + 255) / 256;
    k_adj_cotangent<V><<<(int)(g < 148 * 8 ? g : 148 * 8), 256, 0, s>>>(ybar, (double)T, G, ncomp);
    return cudaGetLastError();
}

cudaError_t launch_adj_scale(CloudCtl* ctl, cudaStream_t s)
{
    k_adj_scale<<<1, 32, 0, s>>>(ctl);
    return cudaGetLastError();
}

cudaError_t launch_adj_mean(const unsigned long long* acc, const CloudCtl* ctl, int limbs,
                            int T, double* mean, int64_t ncomp, cudaStream_t s)
{
    int grid = (int)((ncomp + 255) / 256 < 148 * 8 ? (ncomp + 255) / 256 : 148 * 8);
    if (grid < 1) grid = 1;
    k_adj_mean<<<grid, 256, 0, s>>>(acc, ctl, limbs, (double)T, mean, ncomp);
    return cudaGetLastError();
}

template cudaError_t launch_adj_forward<double, float>(const AdjArgs<double, float>&, bool, cudaStream_t);
template cudaError_t launch_adj_forward<double, double>(const AdjArgs<double, double>&, bool, cudaStream_t);
template cudaError_t launch_adj_reverse<double, float>(const AdjArgs<double, float>&, int, cudaStream_t);
template cudaError_t launch_adj_reverse<double, double>(const AdjArgs<double, double>&, int, cudaStream_t);
template int adj_reverse_grid<double, float>(int64_t, int);
template int adj_reverse_grid<double, double>(int64_t, int);
template cudaError_t launch_adj_cotangent<float>(const double*, int, float*, int64_t, cudaStream_t);
template cudaError_t launch_adj_cotangent<double>(const double*, int, double*, int64_t, cudaStream_t);

}  // namespace st
