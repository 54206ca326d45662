/*
 * st_device.cuh -- device helpers shared by the step kernels of hex (st_kernels.cu) and
 * tetrahedral (st_tet.cu) meshes: IEEE helpers, the fixed-point deterministic deposit with
 * its warp-level run reduction, and the per-warp bookkeeping of the scale tracker.
 */
#ifndef ST_DEVICE_CUH
#define ST_DEVICE_CUH

#include <cstdint>
#include <cuda_runtime.h>

#include "st_internal.h"
#include "st_pow.h"

namespace st {

#ifndef FULL_MASK
#define FULL_MASK 0xffffffffu
#endif

/* Programmatic dependent launch: waits until the kernel before this one on the stream has
 * finished and its writes are visible (at once in a plain launch), and lets the kernel after
 * this one be set up while this one runs. */
__device__ __forceinline__ void grid_dep_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void grid_dep_launch()
{
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ float st_sqrt(float v) { return __fsqrt_rn(v); }
__device__ __forceinline__ double st_sqrt(double v) { return __dsqrt_rn(v); }

__device__ __forceinline__ int32_t st_floor_int(float v) { return __float2int_rd(v); }
__device__ __forceinline__ int32_t st_floor_int(double v) { return __double2int_rd(v); }

/* Slip velocity u_c - v of one component, from the raw cell value Ur and the fluid factor
 * fs = fs_hi + fs_lo.  In mixed precision the product Ur*fs_hi stays exact inside one fma and
 * the low part of the FP64 factor is added, so the slip carries about one rounding of its
 * own size, also when the parcel has nearly relaxed to the carrier (|u - v| << |u|); the
 * FP32 and FP64 modes round u_c = U*fs to the velocity type first, as the reference does
 * (A:1288, A:1295). */
template <bool MIX, class V>
__device__ __forceinline__ V slip(V Ur, V fs_hi, V fs_lo, V vel)
{
    if constexpr (MIX) return __fmaf_rn(Ur, fs_hi, -vel) + Ur * fs_lo;
    else return Ur * fs_hi - vel;
}

/* x^0.687 in single precision (st_pow0687f) with its exponent factor, which depends only on
 * the binary exponent e of x, read from a table in shared memory.  The table is filled on
 * the device by st_pow0687f_efac itself, so the result is st_pow0687f's bit for bit.  A
 * kernel that calls pow0687f_tab fills the table (pow_tab_fill) and synchronises its block
 * first. */
constexpr int POW_TAB_EMIN = -150;   /* st_pow0687f_mant gives -149 <= e <= 128 */
constexpr int POW_TAB_N = 280;
__shared__ float2 s_pow_tab[POW_TAB_N];

__device__ __forceinline__ void pow_tab_fill()
{
    for (int i = threadIdx.x; i < POW_TAB_N; i += blockDim.x) {
        float q, s2k;
        st_pow0687f_efac(i + POW_TAB_EMIN, &q, &s2k);
        s_pow_tab[i] = make_float2(q, s2k);
    }
}

/* Exponent and first factor of st_pow0687f_mant for a positive normal x by integers alone;
 * false for every other x.  With 0x3f3504f4 the float after sqrt(1/2) rounded down, bits -
 * 0x3f3504f4 has the exponent e of x = 2^e m, sqrt(1/2) < m <= sqrt(2), in its upper bits, and
 * subtracting e from the exponent field leaves m. */
__device__ __forceinline__ bool pow0687f_split(float x, int& e, float& p)
{
    const uint32_t b = __float_as_uint(x);
    const int32_t r = (int32_t)(b - 0x3f3504f4u);
    e = r >> 23;
    p = st_pow0687f_poly(__uint_as_float(b - ((uint32_t)r & 0xff800000u)) - 1.0f);
    return b - 0x00800000u < 0x7f000000u;
}

/* st_pow0687f bit for bit: with the table, and with the exponent factor's polynomial */
__device__ __forceinline__ float pow0687f_tab(float x)
{
    int e;
    float p;
    if (!pow0687f_split(x, e, p)) return st_pow0687f(x);   /* 0, subnormal, inf, NaN, < 0 */
    const float2 qs = s_pow_tab[e - POW_TAB_EMIN];
    return (p * qs.x) * qs.y;
}
__device__ __forceinline__ float pow0687f(float x)
{
    int e;
    float p, q, s2k;
    if (!pow0687f_split(x, e, p)) return st_pow0687f(x);
    st_pow0687f_efac(e, &q, &s2k);
    return (p * q) * s2k;
}

/* slip with the product of the raw cell value and the low part of the fluid factor given
 * (Ulo = Ur * fs_lo, formed once per cell by a multi-substep loop): the same value as slip */
template <bool MIX, class V>
__device__ __forceinline__ V slip_lo(V Ur, V fs_hi, V Ulo, V vel)
{
    if constexpr (MIX) return __fmaf_rn(Ur, fs_hi, -vel) + Ulo;
    else return Ur * fs_hi - vel;
}

/* floor(label, v) (A:668-670); values outside int32 mark the parcel as lost.  floor(v) lies
 * in [-2^31, 2^31) exactly when v does (both bounds are integers), so the range test is made
 * on v and one round-down conversion gives the label. */
template <class P>
__device__ __forceinline__ int32_t floor_label(P v, bool& bad)
{
    if (!(v >= (P)-2147483648.0 && v < (P)2147483648.0)) {
        bad = true;
        return 0;
    }
    return st_floor_int(v);
}

/* ------------------------------------------------------------------------------------ */
/* fixed-point deposit                                                                  */
/* ------------------------------------------------------------------------------------ */

/* smallest e with |a| < 2^e, for finite a != 0 (the frexp exponent) */
__device__ __forceinline__ int exp_of(double a)
{
    uint64_t b = (uint64_t)__double_as_longlong(a) & 0x7fffffffffffffffULL;
    int be = (int)(b >> 52);
    if (be == 0) {
        double s = __longlong_as_double((long long)b) * 18014398509481984.0; /* 2^54 */
        be = (int)(((uint64_t)__double_as_longlong(s)) >> 52) - 54;
    }
    return be - 1022;
}

__device__ __forceinline__ double ldexp2(double x, int k)
{
    int k1 = k / 2;
    int k2 = k - k1;
    return (x * st_pow2i(k1)) * st_pow2i(k2);
}

/* The running maximum of |deposit| is kept in the velocity precision (AmaxT<V>): every
 * deposit is a V value, so the maximum is exact in V and needs no conversion per deposit. */
template <class V>
using AmaxT = V;

/* largest finite |v| seen (probe pass) */
__device__ __forceinline__ void track_max(float v, float& amax)
{
    const float a = fabsf(v);
    if (a < __int_as_float(0x7f800000)) amax = fmaxf(amax, a);
}
__device__ __forceinline__ void track_max(double v, double& amax)
{
    const double a = fabs(v);
    if (a < __longlong_as_double(0x7ff0000000000000LL)) amax = fmax(amax, a);
}

/* Fixed-point parameters of one cloud for the current step: q = rint(dep * 2^-L), and a
 * deposit with |dep| >= 2^(cap+L) (i.e. frexp exponent - L > cap) does not fit.  Single
 * precision deposits are scaled in single precision when 2^-L and 2^(cap+L) are normal
 * floats: scaling by a power of two is exact, so the integer is the same as through FP64. */
struct Quant {
    double scale;   /* 2^-L, or 0 when 2^-L is not a normal double (then ldexp2 is used) */
    double thr;     /* 2^(cap+L) */
    float scale_f;  /* 2^-L as float, when `fast` */
    float thr_f;    /* 2^(cap+L) as float, when `fast` */
    int L;
    bool fast;
    float thr_small; /* 2^(SMALL_Q_BITS+L) as float when that is a normal float, else 0 */
};

/* The scale of a step whose largest deposit's exponent a probe has found (EXP_NONE: there is
 * no deposit). */
__device__ __forceinline__ int first_scale(int emax, int H)
{
    return emax == EXP_NONE ? -H : emax - H;
}

/* Quantised deposits below 2^SMALL_Q_BITS in magnitude: a sum of up to eight of them fits in
 * a 32-bit integer (the warp run reduction's 32-bit path). */
constexpr int SMALL_Q_BITS = 28;

__device__ __forceinline__ Quant make_quant(int L, int cap)
{
    Quant q;
    q.L = L;
    q.scale = (-L >= -1022 && -L <= 1023) ? st_pow2i(-L) : 0.0;
    q.thr = ldexp2(1.0, cap + L);
    q.fast = (-L >= -126 && -L <= 127) && (cap + L >= -126 && cap + L <= 127);
    q.scale_f = q.fast ? st_pow2if(-L) : 0.0f;
    q.thr_f = q.fast ? st_pow2if(cap + L) : 0.0f;
    q.thr_small = (q.fast && SMALL_Q_BITS + L >= -126 && SMALL_Q_BITS + L <= 127)
                      ? st_pow2if(SMALL_Q_BITS + L)
                      : 0.0f;
    return q;
}

/* Quantises one deposit component: 0 for zero, non-finite or out-of-range values (the
 * latter two are counted in `ovf`).  `amax` tracks the largest finite |dep| for the next
 * step's scale (max is order-independent, so the scale is reproducible). */
template <class A>
__device__ __forceinline__ long long quantize(double dv, const Quant& qp, A& amax,
                                              unsigned& ovf)
{
    const double a = fabs(dv);
    if (a == 0.0) return 0;
    /* exact for A = float: dv is then a float value */
    if (a < __longlong_as_double(0x7ff0000000000000LL)) amax = (A)fmax((double)amax, a);
    if (!(a < qp.thr)) {
        ++ovf;
        return 0;
    }
    const double x = qp.scale != 0.0 ? dv * qp.scale : ldexp2(dv, -qp.L);
    return __double2ll_rn(x);
}

__device__ __forceinline__ long long quantize(float dv, const Quant& qp, float& amax,
                                              unsigned& ovf)
{
    if (!qp.fast) return quantize((double)dv, qp, amax, ovf);
    const float a = fabsf(dv);
    if (a == 0.0f) return 0;
    if (a < __int_as_float(0x7f800000)) amax = fmaxf(amax, a);
    if (!(a < qp.thr_f)) {
        ++ovf;
        return 0;
    }
    return __float2ll_rn(dv * qp.scale_f);
}

/* The three components of one deposit.  In single precision with the fast scale: when
 * |d0| + |d1| + |d2| (rounded, which cannot fall below a power-of-two bound any single term
 * reaches) is below the range bound, every component is finite and in range, and each is
 * scaled and rounded directly, with the same integers and the same maximum as the
 * per-component path; otherwise (and in double precision) each component goes through
 * quantize, which counts what does not fit. */
__device__ __forceinline__ void quantize3(const float d[3], const Quant& qp, float& amax,
                                          unsigned& ovf, long long q[3])
{
    if (qp.fast) {
        const float a0 = fabsf(d[0]), a1 = fabsf(d[1]), a2 = fabsf(d[2]);
        if ((a0 + a1) + a2 < qp.thr_f) {
            amax = fmaxf(amax, fmaxf(fmaxf(a0, a1), a2));
#pragma unroll
            for (int k = 0; k < 3; ++k) q[k] = __float2ll_rn(d[k] * qp.scale_f);
            return;
        }
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = quantize(d[k], qp, amax, ovf);
}

__device__ __forceinline__ void quantize3(const double d[3], const Quant& qp, double& amax,
                                          unsigned& ovf, long long q[3])
{
#pragma unroll
    for (int k = 0; k < 3; ++k) q[k] = quantize(d[k], qp, amax, ovf);
}

/* Reductions without a return value into global memory.  Spelled out in PTX: where the
 * accumulator's address comes from a descriptor in memory (several clouds in one launch) the
 * compiler sees a generic pointer and issues atomics that return the old value, which each
 * warp then waits for. */
__device__ __forceinline__ void red_add(unsigned long long* p, unsigned long long v)
{
    asm volatile("red.global.add.u64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "l"(v)
                 : "memory");
}
__device__ __forceinline__ void red_add(double* p, double v)
{
    asm volatile("red.global.add.f64 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "d"(v)
                 : "memory");
}

template <int DEP, class V>
__device__ __forceinline__ void deposit_direct(const V dep[3], int64_t cell0,
                                               unsigned long long* acc, double* src,
                                               const Quant& qp, AmaxT<V>& amax, unsigned& ovf)
{
    if constexpr (DEP == DEP_ATOMIC) {
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (dep[c] != (V)0) red_add(src + 3 * cell0 + c, (double)dep[c]);
    } else {
        long long q[3];
        quantize3(dep, qp, amax, ovf, q);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            if (!q[c]) continue;
            if constexpr (DEP == DEP_DET1) {
                red_add(acc + 3 * cell0 + c, (unsigned long long)q[c]);
            } else {
                red_add(acc + 2 * (3 * cell0 + c), (unsigned long long)(q[c] >> 32));
                red_add(acc + 2 * (3 * cell0 + c) + 1, (unsigned long long)q[c] & 0xffffffffULL);
            }
        }
    }
}

/* Steps of the run scan: it sums chunks of 2^steps lanes.  Three steps halve the adds of runs
 * of five to eight parcels against two (a freshly sorted cloud of five parcels per cell); with
 * two limbs a step costs twelve more shuffles, and two steps are faster (FP64, 2e6 parcels on
 * 97 x 64 x 53 cells: 74 us per launch with two steps, 79 us with three and the hand-over of
 * emit_runs). */
template <int DEP>
constexpr int scan_steps = DEP == DEP_DET2 ? 2 : 3;

/* Inclusive scan over the lane's run of equal keys, limited to 2^STEPS lanes (runs are
 * contiguous lane ranges). */
template <int STEPS, class T>
__device__ __forceinline__ T seg_scan(T v, int lane, int segstart)
{
#pragma unroll
    for (int off = 1; off < (1 << STEPS); off <<= 1) {
        T t = __shfl_up_sync(FULL_MASK, v, off);
        if (lane - off >= segstart) v += t;
    }
    return v;
}

/* Streaming loads of the parcel arrays: evict-first (ld.global.cs) so that the cell arrays
 * keep L2, with a 256-byte L2 prefetch hint (each warp reads 128-256 contiguous bytes of an
 * array per tile; measured 0.5 % faster on the 1e7-parcel step than without the hint). */
__device__ __forceinline__ float ld_stream_(const float* p)
{
    float v;
    asm volatile("ld.global.cs.L2::256B.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_stream_(const double* p)
{
    double v;
    asm volatile("ld.global.cs.L2::256B.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int32_t ld_stream_(const int32_t* p)
{
    int32_t v;
    asm volatile("ld.global.cs.L2::256B.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
template <class T>
__device__ __forceinline__ T ld_stream(const T* p) { return ld_stream_(p); }
template <class T>
__device__ __forceinline__ void st_stream(T* p, T v) { __stcs(p, v); }

/* 8-byte words of shared memory, 16-byte aligned, that one warp's deposit_warp needs: up to 96
 * sums and the 32 cells they go to. */
template <int DEP, class V>
constexpr int dep_ws_words = DEP == DEP_ATOMIC                  ? 96 + 16
                             : DEP == DEP_DET1 && sizeof(V) == 4 ? 48 + 16
                                                                 : 1;

/* Writes a warp's run sums out: the lanes with `out` hold three values each (v) for the three
 * consecutive words at dst + 3 * key.  The values are handed over through shared memory so
 * that consecutive lanes add to consecutive words: the words of one cell, and of neighbouring
 * cells, go out in one instruction and merge into few 32-byte sectors, where one instruction
 * per component sends every value as a request of its own.  The adds were what bound the hex
 * step once parcels have drifted from their sorted order (1e7 parcels on 128^3 cells, mean of
 * a re-sort cycle of 20 steps, conversion in stream order: 209 us per launch, 146 us with the
 * adds left out, 186 us with this hand-over and the longer chunks of scan_steps).  The ring hex
 * step writes out with emit_runs_ring instead. */
template <class T, class W>
__device__ __forceinline__ void emit_runs(bool out, int32_t key, const T v[3], W* dst,
                                          unsigned long long* ws, int lane)
{
    const unsigned outs = __ballot_sync(FULL_MASK, out);
    T* const sv = reinterpret_cast<T*>(ws);
    int32_t* const sk = reinterpret_cast<int32_t*>(sv + 96);
    if (out) {
        const int r = __popc(outs & ((1u << lane) - 1u));
#pragma unroll
        for (int k = 0; k < 3; ++k) sv[3 * r + k] = v[k];
        sk[r] = key;
    }
    __syncwarp();
    const int items = 3 * __popc(outs);
    for (int i = lane; i < items; i += 32) {
        const int r = (int)((unsigned)i / 3u);
        const T q = sv[i];
        if (q != (T)0) {
            W* const p = dst + 3 * (int64_t)sk[r] + (i - 3 * r);
            if constexpr (sizeof(T) == 4) red_add(p, (W)(long long)q);
            else red_add(p, (W)q);
        }
    }
    __syncwarp();
}

/* emit_runs for the 32-bit sums of the ring hex step with one substep, which every instruction
 * counts in.  The sums go to shared memory with their cell in one 16-byte store.
 *
 * `emit` is what the warp found at the first sums it wrote that were not all zero.  In a planar
 * flow no sum has three non-zero components, there are a third fewer adds, and direct ones, one
 * instruction per component, are faster.  1e7 parcels on 128^3 cells from rest, conversion
 * overlapped, us per step over 20, 100 and 500 steps: without a z component 223 / 224 / 224
 * handed over, 221 / 219 / 217 by this rule, 216 / 216 / 215 added directly in a kernel that has
 * no other way; with three components 226 / 227 handed over and by this rule, 249 direct.
 * (The vote on every call costs the second flow 1 to 2 %; an instance of the whole tile for
 * each of the two, 5 %.) */
enum Emit { EMIT_UNKNOWN = 0, EMIT_HAND_OVER = 1, EMIT_DIRECT = 2 };

__device__ __forceinline__ void emit_runs_ring(bool out, int32_t key, const int v[3],
                                               unsigned long long* acc, unsigned long long* ws,
                                               int lane, int& emit)
{
    if (emit == EMIT_UNKNOWN) {
        const int nz = out ? (v[0] != 0) + (v[1] != 0) + (v[2] != 0) : 0;
        const int most = __reduce_max_sync(FULL_MASK, nz);
        if (most) emit = most == 3 ? EMIT_HAND_OVER : EMIT_DIRECT;
    }
    if (emit == EMIT_DIRECT) {
        if (out) {
            unsigned long long* const p = acc + 3 * (int64_t)key;
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (v[k]) red_add(p + k, (unsigned long long)(long long)v[k]);
        }
        return;
    }
    const unsigned outs = __ballot_sync(FULL_MASK, out);
    if (out)
        reinterpret_cast<int4*>(ws)[__popc(outs & ((1u << lane) - 1u))] =
            make_int4(v[0], v[1], v[2], key);
    __syncwarp();
    const int items = 3 * __popc(outs);
    const int* const s = reinterpret_cast<const int*>(ws);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const int i = lane + 32 * t;
        if (i < items) {
            const int r = (i * 43) >> 7;   /* i / 3, exact for i < 128 */
            const int q = s[i + r];
            unsigned long long* const p = acc + (3 * (int64_t)s[4 * r + 3] + (i - 3 * r));
            if (q) red_add(p, (unsigned long long)(long long)q);
        }
    }
    __syncwarp();
}

/* Final deposits of 32 consecutive parcels (one per lane, key < 0 = none): runs of equal
 * cells are summed with a segmented warp scan and the last lane of each run adds the sum.
 * The FP64 atomic mode sums its runs in FP64 the same way.
 * `ws`: this warp's dep_ws_words<DEP, V> words of shared memory.  `emit`: emit_runs_ring's, for
 * its caller. */
template <int DEP, class V>
__device__ __forceinline__ void deposit_warp(int32_t key, const V dep[3],
                                             unsigned long long* acc, double* src,
                                             const Quant& qp, int lane, AmaxT<V>& amax,
                                             unsigned& ovf, unsigned long long* ws,
                                             int* emit = nullptr)
{
    if (DEP == DEP_PROBE) {
        if (key >= 0) {
#pragma unroll
            for (int k = 0; k < 3; ++k) track_max(dep[k], amax);
        }
        return;
    }
    constexpr int STEPS = scan_steps<DEP>, SPAN = 1 << STEPS;
    const int prev = __shfl_up_sync(FULL_MASK, key, 1);
    const bool head = (lane == 0) || (prev != key);
    const unsigned heads = __ballot_sync(FULL_MASK, head);
    /* quantised deposits, and whether the 32-bit path holds for every lane */
    int q32[3] = {0, 0, 0};
    bool narrow = false;
    if constexpr (DEP == DEP_DET1 && sizeof(V) == 4) {
        /* 32-bit path: when every lane's deposit components quantise below 2^SMALL_Q_BITS
         * (|d0| + |d1| + |d2| below 2^(SMALL_Q_BITS+L), the bound argument of quantize3), the
         * integers are those of quantize3, a chunk of SPAN <= 8 lanes sums below 2^31, and the
         * run sums are formed in 32-bit registers: the same integers reach the accumulators. */
        bool small = key < 0;
        if (key >= 0) {
            const float a0 = fabsf((float)dep[0]), a1 = fabsf((float)dep[1]),
                        a2 = fabsf((float)dep[2]);
            if ((a0 + a1) + a2 < qp.thr_small) {
                amax = fmaxf(amax, fmaxf(fmaxf(a0, a1), a2));
#pragma unroll
                for (int k = 0; k < 3; ++k) q32[k] = __float2int_rn((float)dep[k] * qp.scale_f);
                small = true;
            }
        }
        static_assert(SMALL_Q_BITS + STEPS <= 31, "32-bit chunk sums");
        narrow = __all_sync(FULL_MASK, small);
        if (narrow && heads == 1u) {
            /* one cell for the whole warp: 16-bit halves, each sum exact in 32 bits */
            if (key >= 0) {
                long long t[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int shi = __reduce_add_sync(FULL_MASK, q32[k] >> 16);
                    const unsigned slo = __reduce_add_sync(FULL_MASK, (unsigned)q32[k] & 0xffffu);
                    t[k] = (long long)shi * 65536LL + (long long)slo;
                }
                const long long mine = lane == 0 ? t[0] : (lane == 1 ? t[1] : t[2]);
                if (lane < 3 && mine)
                    red_add(acc + 3 * (int64_t)key + lane, (unsigned long long)mine);
            }
            return;
        }
    }
    long long q[3] = {0, 0, 0};
    if constexpr (DEP != DEP_ATOMIC) {
        if (!narrow && key >= 0) quantize3(dep, qp, amax, ovf, q);
    }
    if (DEP == DEP_DET1 && !narrow && heads == 1u) {
        /* One cell for the whole warp (dense cells after a re-sort): exact full-warp
         * reductions replace the scan.  With q = hi*2^32 + lo, the sums of lo's two 16-bit
         * halves stay below 2^21, and |sum of hi| <= 2^30 + 32 because the headroom bounds
         * the magnitudes of all of a step's deposits together by 2^62. */
        if (key >= 0) {
            long long t[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const unsigned lo = (unsigned)(unsigned long long)q[k];
                const long long shi = __reduce_add_sync(FULL_MASK, (int)(q[k] >> 32));
                const unsigned s0 = __reduce_add_sync(FULL_MASK, lo & 0xffffu);
                const unsigned s1 = __reduce_add_sync(FULL_MASK, lo >> 16);
                t[k] = shi * 4294967296LL + (long long)s0 + (long long)s1 * 65536LL;
            }
            const long long mine = lane == 0 ? t[0] : (lane == 1 ? t[1] : t[2]);
            if (lane < 3 && mine)
                red_add(acc + 3 * (int64_t)key + lane, (unsigned long long)mine);
        }
        return;
    }
    /* A scan of STEPS steps sums runs in chunks of SPAN lanes: lane j holds the sum of
     * [max(run start, j - SPAN + 1), j]; the run's last lane and every SPAN-th lane before it
     * add their chunk, which covers the run exactly once. */
    const int segstart = 31 - __clz(heads & (FULL_MASK >> (31 - lane)));
    const bool tail = (lane == 31) || ((heads >> (lane + 1)) & 1u);
    const unsigned tails = __ballot_sync(FULL_MASK, tail);
    const int tailpos = lane + __ffs(tails >> lane) - 1;
    const bool out = ((tailpos - lane) & (SPAN - 1)) == 0 && key >= 0;
    if constexpr (DEP == DEP_ATOMIC) {
        double t[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = seg_scan<STEPS>((double)dep[k], lane, segstart);
        emit_runs(out, key, t, src, ws, lane);
    } else if constexpr (DEP == DEP_DET1) {
        if (narrow) {
#pragma unroll
            for (int k = 0; k < 3; ++k) q32[k] = seg_scan<STEPS>(q32[k], lane, segstart);
            if (emit) emit_runs_ring(out, key, q32, acc, ws, lane, *emit);
            else emit_runs(out, key, q32, acc, ws, lane);
            return;
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) q[k] = seg_scan<STEPS>(q[k], lane, segstart);
        if (out) {   /* a warp with a large deposit, or FP32 deposits outside the fast range */
            unsigned long long* p = acc + 3 * (int64_t)key;
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (q[k]) red_add(p + k, (unsigned long long)q[k]);
        }
    } else {
        long long hi[3];
        unsigned long long lo[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            hi[k] = seg_scan<STEPS>(q[k] >> 32, lane, segstart);
            lo[k] = seg_scan<STEPS>((unsigned long long)q[k] & 0xffffffffULL, lane, segstart);
        }
        if (out) {
            unsigned long long* p = acc + 6 * (int64_t)key;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (hi[k]) red_add(p + 2 * k, (unsigned long long)hi[k]);
                if (lo[k]) red_add(p + 2 * k + 1, lo[k]);
            }
        }
    }
}

/* Warp-aggregated bookkeeping for one cloud: largest deposit exponent, lost parcels and
 * range errors.  Called when a warp moves on to another cloud and at the end. */
template <int DEP, class A>
__device__ __forceinline__ void flush_ctl(CloudCtl* ctl, int lane, A& amax, unsigned& ovf,
                                          unsigned& lost, int* block_emax = nullptr)
{
    /* block_emax (shared memory): the warp's largest exponent goes there, and the kernel adds
     * the block's maximum to the control block once */
    if (DEP != DEP_ATOMIC) {
        const int e = amax > (A)0 ? exp_of((double)amax) : EXP_NONE;
        const int wmax = __reduce_max_sync(FULL_MASK, e);
        if (lane == 0 && wmax != EXP_NONE) atomicMax(block_emax ? block_emax : &ctl->emax, wmax);
    }
    const unsigned nlost = __reduce_add_sync(FULL_MASK, lost);
    const unsigned novf = __reduce_add_sync(FULL_MASK, ovf);
    if (lane == 0) {
        /* the probe pass repeats the step: only the real pass reports */
        if (nlost && DEP != DEP_PROBE) atomicAdd(&ctl->lost, (unsigned long long)nlost);
        if (novf && DEP != DEP_PROBE) atomicAdd(&ctl->overflow, (unsigned long long)novf);
    }
    amax = (A)0;
    ovf = 0;
    lost = 0;
}

}  // namespace st

#endif
