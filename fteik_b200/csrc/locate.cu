/*
 * locate.cu -- grid-search event location (locate.F90:620-744, :112-126).
 *
 * fk_locate_l2_exact reproduces the reference's FP32 objective bit for bit:
 * for every grid point g and event e, in the reference's order,
 *   t0[g]  += w_i * (xnorm * (o_i - T_i[g]))            over used tables i
 *   obj[g] += ((sqrt(1/2) * w_i) * (o_i - (T_i[g] + t0[g])))^2
 * with no fused multiply-add, then MINLOC (first minimum).  A thread keeps
 * the tables of its grid points in registers and evaluates the events
 * against them, so the tables stream from HBM once per CTA rather than once
 * per event.  The argmin is a 64-bit atomicMin on (float bits of obj) << 32
 * | g, which for non-negative objectives orders by value and then by the
 * smaller index, as MINLOC does.
 *
 * Most points are ruled out before the objective is evaluated there
 * (l2_search_kernel<NTF, true>): for any subset A of the picks and any t0,
 *   2 obj >= min_t sum_A w^2 (o - T - t)^2 = s2 - s3^2 / sum_A w^2,
 *   s2 = sum_A (w (o - T))^2,  s3 = sum_A w^2 (o - T),
 * three multiply-adds a pick instead of the objective's nine operations.
 * A point is skipped only if this bound, less the rounding errors of both
 * sides, exceeds the event's best objective so far, so the optimum, its
 * index and its ties are those of the full search.  The first best value
 * comes from a strided sample of the points.
 */
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include "fteik_dev.h"

namespace {

constexpr int kMaxTf = 64;    /* tables held in registers */
constexpr int kThreads = 128; /* 4 warps of 64 points (L2) or 32 points (L1) */
constexpr int kEvChunk = 16;  /* events staged in shared memory at a time */
constexpr int kLevels = 8;    /* the bound's subsets: tables l, l + 8, l + 16, ... are level l's */

__device__ __forceinline__ unsigned long long pack_key(float obj, int g)
{
    return ((unsigned long long)__float_as_uint(obj) << 32) | (unsigned)g;
}

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

__device__ __forceinline__ unsigned long long warp_min(unsigned long long key)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long k2 = __shfl_xor_sync(0xffffffffu, key, o);
        key = k2 < key ? k2 : key;
    }
    return key;
}

/* Rounding allowances of the L2 bound, e = 2^-24, k <= 64 picks.  With O2 =
 * sum (w o)^2 over the event's picks, the computed s2 - s3^2 / sum w^2 is at
 * most (3 k + 9) e s2 + 2 e O2 above the exact one (each w (o - T) is one
 * multiply-add of a rounded w o), and the reference's objective at most
 * (k + 16) e obj + e O2 / 2 below the exact misfit at its own t0. */
constexpr float kSlackS2 = 1.0f / 65536;   /* 2^-16 >= (3 k + 32) e */
constexpr float kSlackObj = 1.0f / 65536;  /* 2^-16 >= (k + 36) e */
constexpr float kSlackO2 = 1.0f / 1048576; /* 2^-20 = 16 e */

/* Searches the points p stride, p < np = ceil(ngrd / stride).  A warp owns 64
 * points, two per lane (32 apart, so every load is 4-byte and coalesced
 * whatever the tables' alignment) in packed FP32 arithmetic.  A CTA keeps its
 * tables while it runs over the events blockIdx.y, + gridDim.y, ... (in
 * chunks of kEvChunk).  BOUND: rule out by the bound first, level by level
 * (the sums carry on), while any of the warp's points survives.  The bound
 * costs 3 packed operations and one 16-byte shared-memory broadcast a pick. */
template <int NTF, bool BOUND>
__global__ void __launch_bounds__(kThreads, NTF == 64 ? 3 : 4)
l2_search_kernel(int ngrd, int ldgrd, int ntf, int stride, const float *__restrict__ tables, int nev,
                 const float *__restrict__ obs, const float *__restrict__ wts,
                 const float *__restrict__ xnorm, unsigned long long *best)
{
    __shared__ float4 s_lb[BOUND ? kEvChunk : 1][NTF];   /* w, w, w o, w o */
    __shared__ float2 s_ow[kEvChunk][NTF];
    __shared__ float s_is2[kEvChunk][kLevels], s_o2[kEvChunk], s_xn[kEvChunk];
    __shared__ unsigned s_u[kEvChunk];                   /* float bits of the best objective so far */
    __shared__ unsigned long long s_best[kEvChunk];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long p0 = ((long long)blockIdx.x * (kThreads / 32) + warp) * 64 + lane;
    const long long gl0 = p0 * stride, gl1 = (p0 + 32) * stride;
    const bool in0 = gl0 < ngrd, in1 = gl1 < ngrd;
    const int g0 = in0 ? (int)gl0 : 0, g1 = in1 ? (int)gl1 : 0;
    float2 nT[NTF];                                      /* -T of the two points */
#pragma unroll
    for (int i = 0; i < NTF; ++i) {
        float a = 0.0f, b = 0.0f;
        if (i < ntf && in0) a = __ldg(tables + (size_t)i * ldgrd + g0);
        if (i < ntf && in1) b = __ldg(tables + (size_t)i * ldgrd + g1);
        nT[i] = make_float2(-a, -b);
    }
    const int nchunk = (nev + kEvChunk - 1) / kEvChunk;
    for (int c = blockIdx.y; c < nchunk; c += gridDim.y) {
        const int e0 = c * kEvChunk, nb = min(kEvChunk, nev - e0);
        __syncthreads();
#pragma unroll 1
        for (int t = threadIdx.x; t < kEvChunk * NTF; t += kThreads) {
            const int e = t / NTF, i = t % NTF;
            float o = 0.0f, w = 0.0f;
            if (e < nb && i < ntf) {
                w = wts[(size_t)(e0 + e) * ntf + i];
                o = obs[(size_t)(e0 + e) * ntf + i];
                if (!(w > 0.0f)) o = w = 0.0f;           /* a skipped pick */
            }
            s_ow[e][i] = make_float2(o, w);
            if (BOUND) s_lb[e][i] = make_float4(w, w, w * o, w * o);
        }
        __syncthreads();
#pragma unroll 1
        for (int e = warp; e < nb; e += kThreads / 32) { /* per event: the levels' 1 / sum w^2, and O2 */
            float a = 0.0f, o2 = 0.0f;
            for (int i = lane; i < NTF; i += 32) {       /* lane mod 8 = level */
                const float2 ow = s_ow[e][i];
                a += ow.y * ow.y;
                o2 += (ow.x * ow.y) * (ow.x * ow.y);
            }
            if (NTF < 32 && lane >= NTF) a = o2 = 0.0f;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) o2 += __shfl_xor_sync(0xffffffffu, o2, o);
#pragma unroll
            for (int o = 16; o >= kLevels; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
            /* inclusive over the levels: lane l holds levels 0 .. l */
            float up = __shfl_up_sync(0xffffffffu, a, 1);
            if (lane >= 1) a += up;
            up = __shfl_up_sync(0xffffffffu, a, 2);
            if (lane >= 2) a += up;
            up = __shfl_up_sync(0xffffffffu, a, 4);
            if (lane >= 4) a += up;
            if (lane < kLevels) s_is2[e][lane] = a > 0.0f ? 1.0f / a : 0.0f;
            if (lane == 0) {
                s_o2[e] = kSlackO2 * o2;
                s_xn[e] = xnorm[e0 + e];
                const unsigned long long b = __ldcg(best + e0 + e);
                s_u[e] = (unsigned)(b >> 32);            /* none yet: a NaN, which rules nothing out */
                s_best[e] = ~0ull;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int e = 0; e < nb; ++e) {
            if (BOUND) {
                const float u = __uint_as_float(*(volatile unsigned *)&s_u[e]);
                const float thr = fmaf(2.0f * u, 1.0f + kSlackObj, s_o2[e]);
                float2 s2a = dup(0.0f), s2b = s2a, s3a = s2a, s3b = s2a;
                bool any = true;
#pragma unroll
                for (int l = 0; l < kLevels; ++l) {
#pragma unroll
                    for (int i = l; i < NTF; i += 2 * kLevels) {
                        const float4 q = s_lb[e][i];
                        const float2 w = make_float2(q.x, q.y);
                        const float2 p = __ffma2_rn(w, nT[i], make_float2(q.z, q.w));
                        s2a = __ffma2_rn(p, p, s2a);
                        s3a = __ffma2_rn(w, p, s3a);
                        const float4 q2 = s_lb[e][i + kLevels];
                        const float2 w2 = make_float2(q2.x, q2.y);
                        const float2 p2 = __ffma2_rn(w2, nT[i + kLevels], make_float2(q2.z, q2.w));
                        s2b = __ffma2_rn(p2, p2, s2b);
                        s3b = __ffma2_rn(w2, p2, s3b);
                    }
                    const float2 s2 = __fadd2_rn(s2a, s2b), s3 = __fadd2_rn(s3a, s3b);
                    const float2 m = __fmul2_rn(s3, dup(-s_is2[e][l]));
                    const float2 lb = __ffma2_rn(m, s3, __ffma2_rn(s2, dup(-kSlackS2), s2));
                    any = __any_sync(0xffffffffu, (in0 && !(lb.x > thr)) || (in1 && !(lb.y > thr)));
                    if (!any) break;
                }
                if (!any) continue;
            }
            const float2 xn = dup(s_xn[e]);
            float2 t0 = dup(0.0f);
#pragma unroll
            for (int i = 0; i < NTF; ++i) {
                const float2 ow = s_ow[e][i];
                if (ow.y > 0.0f) {
                    const float2 res = __fmul2_rn(xn, __fadd2_rn(dup(ow.x), nT[i]));
                    t0 = __fadd2_rn(t0, __fmul2_rn(dup(ow.y), res));
                }
            }
            const float2 nt0 = make_float2(-t0.x, -t0.y);
            float2 obj = dup(0.0f);
#pragma unroll
            for (int i = 0; i < NTF; ++i) {
                /* read again (volatile): kept from the first pass, the picks alone are 128 registers */
                const unsigned long long q = *(volatile const unsigned long long *)&s_ow[e][i];
                const float2 ow = make_float2(__uint_as_float((unsigned)q), __uint_as_float((unsigned)(q >> 32)));
                if (ow.y > 0.0f) {
                    const float wt = __fmul_rn(0.70710677f, ow.y); /* SQRT(0.5) in FP32 (constants.F90) */
                    const float2 res = __fmul2_rn(dup(wt), __fadd2_rn(dup(ow.x), __fadd2_rn(nT[i], nt0)));
                    obj = __fadd2_rn(obj, __fmul2_rn(res, res));
                }
            }
            unsigned long long key = in0 ? pack_key(obj.x, g0) : ~0ull;
            const unsigned long long k1 = in1 ? pack_key(obj.y, g1) : ~0ull;
            key = warp_min(k1 < key ? k1 : key);
            if (lane == 0) {
                atomicMin(&s_best[e], key);
                atomicMin(&s_u[e], (unsigned)(key >> 32));
            }
        }
        __syncthreads();
        if (threadIdx.x < nb && s_best[threadIdx.x] != ~0ull) atomicMin(best + e0 + threadIdx.x, s_best[threadIdx.x]);
    }
}

/* t0 and obj at the optimum, same arithmetic: a warp per event fetches its
 * 64 terms at once, one lane adds them in order. */
__global__ void __launch_bounds__(128)
l2_at_opt_kernel(int ldgrd, int ntf, const float *__restrict__ tables, int nev, const float *__restrict__ obs,
                 const float *__restrict__ wts, const float *__restrict__ xnorm,
                 const unsigned long long *__restrict__ best, int *out_idx, float *out_t0, float *out_obj)
{
    __shared__ float s_o[4][kMaxTf], s_w[4][kMaxTf], s_t[4][kMaxTf];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.x * 4 + warp;
    if (e >= nev) return;
    const int g = (int)(best[e] & 0xffffffffu);
    for (int i = lane; i < ntf; i += 32) {
        s_o[warp][i] = obs[(size_t)e * ntf + i];
        s_w[warp][i] = wts[(size_t)e * ntf + i];
        s_t[warp][i] = tables[(size_t)i * ldgrd + g];
    }
    __syncwarp();
    if (lane != 0) return;
    const float *o = s_o[warp], *w = s_w[warp], *T = s_t[warp];
    const float xn = xnorm[e];
    float t0 = 0.0f;
    for (int i = 0; i < ntf; ++i)
        if (w[i] > 0.0f) t0 = __fadd_rn(t0, __fmul_rn(w[i], __fmul_rn(xn, __fsub_rn(o[i], T[i]))));
    float obj = 0.0f;
    for (int i = 0; i < ntf; ++i)
        if (w[i] > 0.0f) {
            const float res = __fmul_rn(__fmul_rn(0.70710677f, w[i]), __fsub_rn(o[i], __fadd_rn(T[i], t0)));
            obj = __fadd_rn(obj, __fmul_rn(res, res));
        }
    out_idx[e] = g;
    out_t0[e] = t0;
    out_obj[e] = obj;
}

__global__ void xnorm_kernel(int nev, int ntf, const float *__restrict__ wts, float *xnorm,
                             unsigned long long *best)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nev) return;
    float s = 0.0f; /* SUM over the padded weight row, in order */
    for (int i = 0; i < ntf; ++i) s = __fadd_rn(s, wts[(size_t)e * ntf + i]);
    xnorm[e] = __fdiv_rn(1.0f, s);
    best[e] = ~0ull;
}

/* Searches the points in one launch, or in two: fewer than kBoundEvents
 * events are bound by reading the tables once, and a few thousand points by
 * the launches, so there every point is evaluated; from there on a sample of
 * every kSample-th point sets the best values that the bound needs.  512
 * events x 64 tables x 2.46e6 points: 6.8, 6.5 and 6.5 ms with every 128th,
 * 256th and 512th point (4 levels instead of 8: 4 % more), 100.5 ms with the
 * objective evaluated everywhere and its skipped picks predicated; 60 events
 * x 20 tables x 168,000 points: 118 us against 303. */
constexpr int kBoundEvents = 8, kBoundPoints = 4096;
constexpr int kSample = 256;

/* CTAs over the events when the points alone leave the chip idle (148 SMs,
 * 3 CTAs each, a few waves) */
inline int event_split(long long ctas, int nev)
{
    const int nchunk = (nev + kEvChunk - 1) / kEvChunk;
    long long y = (148 * 3 * 4 + ctas - 1) / ctas;
    return (int)(y < 1 ? 1 : y > nchunk ? nchunk : y);
}

template <int NTF>
void launch_l2_search(int ngrd, int ldgrd, int ntf, const float *tables, int nev, const float *obs, const float *wts,
                      const float *xn, unsigned long long *best, cudaStream_t s)
{
    const int per = kThreads / 32 * 64;
    const long long ctas = (ngrd + (long long)per - 1) / per;
    const dim3 grid((unsigned)ctas, event_split(ctas, nev));
    if (nev < kBoundEvents || ngrd < kBoundPoints) {
        l2_search_kernel<NTF, false><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, obs, wts, xn, best);
        return;
    }
    const long long cs = ((ngrd + kSample - 1) / kSample + (long long)per - 1) / per;
    l2_search_kernel<NTF, false><<<dim3((unsigned)cs, event_split(cs, nev)), kThreads, 0, s>>>(
        ngrd, ldgrd, ntf, kSample, tables, nev, obs, wts, xn, best);
    l2_search_kernel<NTF, true><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, obs, wts, xn, best);
}

} // namespace

extern "C" size_t fk_locate_l2_exact_scratch(int ngrd, int nev)
{
    (void)ngrd;
    return (size_t)nev * (sizeof(unsigned long long) + sizeof(float)) + 256;
}

extern "C" int fk_locate_l2_exact(int ngrd, int ldgrd, int ntf, const float *tables, int nev,
                                  const float *obs, const float *wts, int *out_idx,
                                  float *out_t0, float *out_obj, void *scratch,
                                  size_t scratch_bytes, cudaStream_t s)
{
    if (nev <= 0) return 0;
    if (ntf > kMaxTf || ntf < 1) return (int)cudaErrorInvalidValue;
    if (scratch_bytes < fk_locate_l2_exact_scratch(ngrd, nev)) return (int)cudaErrorInvalidValue;
    unsigned long long *best = (unsigned long long *)scratch;
    float *xn = (float *)(best + nev);
    xnorm_kernel<<<(nev + 127) / 128, 128, 0, s>>>(nev, ntf, wts, xn, best);
    if (ntf <= 16) launch_l2_search<16>(ngrd, ldgrd, ntf, tables, nev, obs, wts, xn, best, s);
    else if (ntf <= 32) launch_l2_search<32>(ngrd, ldgrd, ntf, tables, nev, obs, wts, xn, best, s);
    else launch_l2_search<64>(ngrd, ldgrd, ntf, tables, nev, obs, wts, xn, best, s);
    l2_at_opt_kernel<<<(nev + 3) / 4, 128, 0, s>>>(ldgrd, ntf, tables, nev, obs, wts, xn, best, out_idx, out_t0,
                                                   out_obj);
    return (int)cudaGetLastError();
}

/* ------------------------------------------------------------------------ */
/* Allocation-free variant.                                                 */
/*                                                                          */
/* Some callers cannot let a library call cudaMalloc: a host that hands out */
/* all device memory from its own pool (a framework's caching allocator, a  */
/* real-time service with a fixed memory budget) or that must not trigger   */
/* the device-wide synchronisation cudaMalloc/cudaFree can cause.  For them */
/* fteik_b200_locate_l2_noalloc runs the same grid search on buffers the    */
/* caller owns, keeping its per-event scratch (the best (misfit, index) key */
/* and the weight normaliser, 12 bytes per event) in the fixed array below. */
/* ------------------------------------------------------------------------ */

#define FK_NOALLOC_MAX_EVENTS 65536
/* Lives on every device that loads this library until the process exits. */
static __device__ __align__(256) unsigned char g_noalloc_scratch[FK_NOALLOC_MAX_EVENTS * 12 + 256];

extern "C" void fteik_b200_locate_l2_noalloc(int ngrd, int ldgrd, int ntf, const float *tables,
                                             int nev, const float *obs, const float *wts,
                                             int *opt_index, float *t0, float *obj, void *stream,
                                             int *ierr)
{
    *ierr = 1;
    if (nev < 1 || nev > FK_NOALLOC_MAX_EVENTS) {
        fprintf(stderr, "fteik_b200_locate_l2_noalloc: nev=%d must be in [1,%d]\n", nev,
                FK_NOALLOC_MAX_EVENTS);
        return;
    }
    if (ntf < 1 || ntf > kMaxTf || ngrd < 1 || ldgrd < ngrd) {
        fprintf(stderr, "fteik_b200_locate_l2_noalloc: need 1 <= ntf <= %d and 1 <= ngrd <= ldgrd\n",
                kMaxTf);
        return;
    }
    if (!tables || !obs || !wts || !opt_index || !t0 || !obj) {
        fprintf(stderr, "fteik_b200_locate_l2_noalloc: null buffer\n");
        return;
    }
    /* the device address of the array, looked up on every call with the
     * caller's current device (the host-side name of the array is not a
     * device address); nothing is cached, so concurrent first calls from
     * several host threads and a reset device leave no stale address */
    void *scratch = NULL;
    cudaError_t e = cudaGetSymbolAddress(&scratch, g_noalloc_scratch);
    if (e != cudaSuccess) {
        fprintf(stderr, "fteik_b200_locate_l2_noalloc: cudaGetSymbolAddress failed (%s)\n",
                cudaGetErrorString(e));
        return;
    }
    const int rc = fk_locate_l2_exact(ngrd, ldgrd, ntf, tables, nev, obs, wts, opt_index, t0, obj,
                                      scratch, sizeof(g_noalloc_scratch),
                                      (cudaStream_t)stream);
    if (rc != 0) {
        fprintf(stderr, "fteik_b200_locate_l2_noalloc: launch failed (%s)\n",
                cudaGetErrorString((cudaError_t)rc));
        return;
    }
    *ierr = 0;
}

/* ------------------------------------------------------------------------ */
/* L1 grid search (no counterpart in the reference, which has L2 only).     */
/*                                                                          */
/* For the picks of an event (positive weights, all equal to w) and a grid  */
/* point g the residuals r_i = o_i - T_i(g) give                            */
/*   t0(g)  = median of r  (any point between the two middle values when   */
/*            the count is even; the midpoint is reported)                  */
/*   obj(g) = w sum_i |r_i - t0| = w (sum of the upper half - sum of the    */
/*            lower half of the sorted residuals).                          */
/* A thread holds the 64 residuals of one grid point in registers and sorts */
/* them with a fully unrolled bitonic network (skipped picks sort last as   */
/* +inf); the half sums use compile-time indices.  Most points are ruled    */
/* out first by a bound on the misfit (l1_search_kernel).  The argmin is    */
/* the first-index minimum (64-bit atomicMin on (bits << 32) | g); t0 and   */
/* obj at the optimum are recomputed in FP64.                               */
/* ------------------------------------------------------------------------ */

namespace {

template <int N>
__device__ __forceinline__ void bitonic_sort(float (&v)[N])
{
#pragma unroll
    for (int k = 2; k <= N; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1)
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const int l = i ^ j;
                if (l > i) {
                    const float a = v[i], b = v[l];
                    const bool up = (i & k) == 0;
                    v[i] = up ? fminf(a, b) : fmaxf(a, b);
                    v[l] = up ? fmaxf(a, b) : fminf(a, b);
                }
            }
}

/* Rounding allowance of the L1 bound: with e = 2^-24 the ranking misfit is
 * computed to (N + 1) e sum (|o| + |T|) and the pairs' sum to (N / 2 + 4) e of
 * the same, N <= 64 (times the event's weight). */
constexpr float kSlackL1 = 1.0f / 131072;   /* 2^-17 = 128 e */

/* Searches the points p stride; a warp owns 32 points, one a lane, and runs
 * over the events as l2_search_kernel does.  BOUND: for any t0 two picks
 * give |r_i - t0| + |r_j - t0| >= |r_i - r_j|, so the sum over disjoint pairs
 * (i, i + N / 2) bounds the misfit from below at four operations a pair,
 * against the sorting network's 672 compare-exchanges for 64 picks; the
 * pairs come in kLevels levels, and a point is sorted only if all of them
 * stay below the event's best misfit so far.  A pair with a skipped pick
 * counts zero (its cap).  128 events x 64 tables x 2.46e6 points: 3.3 ms
 * (3.7 and 3.4 ms with every 64th and 1024th point in the sample) against
 * 38.6 ms with every point sorted. */
template <int N, bool BOUND>
__global__ void __launch_bounds__(kThreads, 3)
l1_search_kernel(int ngrd, int ldgrd, int ntf, int stride, const float *__restrict__ tables, int nev,
                 const float *__restrict__ obs, const float *__restrict__ wts, unsigned long long *best)
{
    __shared__ float s_obs[kEvChunk][N];
    __shared__ float s_w[kEvChunk][N];
    __shared__ float2 s_pair[BOUND ? kEvChunk : 1][N / 2];   /* o_i - o_j, cap */
    __shared__ int s_n[kEvChunk];
    __shared__ float s_wv[kEvChunk], s_o[kEvChunk];
    __shared__ unsigned s_u[kEvChunk];                       /* float bits of the best misfit so far */
    __shared__ unsigned long long s_best[kEvChunk];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long gl = ((long long)blockIdx.x * kThreads + threadIdx.x) * stride;
    const bool in = gl < ngrd;
    const int g = in ? (int)gl : 0;
    const float INF = __int_as_float(0x7f800000);
    float T[N], sumT = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        T[i] = (in && i < ntf) ? __ldg(tables + (size_t)i * ldgrd + g) : 0.0f;
        sumT += fabsf(T[i]);
    }
    const int nchunk = (nev + kEvChunk - 1) / kEvChunk;
    for (int c = blockIdx.y; c < nchunk; c += gridDim.y) {
        const int e0 = c * kEvChunk, nb = min(kEvChunk, nev - e0);
        __syncthreads();
#pragma unroll 1
        for (int t = threadIdx.x; t < kEvChunk * N; t += kThreads) {
            const int e = t / N, i = t % N;
            const bool ok = e < nb && i < ntf;
            s_obs[e][i] = ok ? obs[(size_t)(e0 + e) * ntf + i] : 0.0f;
            s_w[e][i] = ok ? wts[(size_t)(e0 + e) * ntf + i] : 0.0f;
        }
        __syncthreads();
#pragma unroll 1
        for (int e = warp; e < nb; e += kThreads / 32) {
            int n = 0;
            float wv = 0.0f, so = 0.0f;
            for (int i = lane; i < N; i += 32)
                if (s_w[e][i] > 0.0f) { ++n; wv = s_w[e][i]; so += fabsf(s_obs[e][i]); }
            if (BOUND)
                for (int i = lane; i < N / 2; i += 32)
                    s_pair[e][i] = make_float2(s_obs[e][i] - s_obs[e][i + N / 2],
                                               s_w[e][i] > 0.0f && s_w[e][i + N / 2] > 0.0f ? INF : 0.0f);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                n += __shfl_xor_sync(0xffffffffu, n, o);
                wv = fmaxf(wv, __shfl_xor_sync(0xffffffffu, wv, o));   /* one weight per event */
                so += __shfl_xor_sync(0xffffffffu, so, o);
            }
            if (lane == 0) {
                s_n[e] = n;
                s_wv[e] = wv;
                s_o[e] = so;
                const unsigned long long b = __ldcg(best + e0 + e);
                s_u[e] = (unsigned)(b >> 32);                /* none yet: a NaN, which rules nothing out */
                s_best[e] = ~0ull;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int e = 0; e < nb; ++e) {
            if (BOUND) {
                const float u = __uint_as_float(*(volatile unsigned *)&s_u[e]);
                /* a misfit of -0 or rounded below zero orders after all others (its key is unsigned) */
                const float thr = signbit(u) ? INF
                                             : fmaf(u / s_wv[e], 1.0f + 1.0f / 1048576, kSlackL1 * (sumT + s_o[e]));
                float la = 0.0f;
                bool any = true;
#pragma unroll
                for (int l = 0; l < kLevels; ++l) {
#pragma unroll
                    for (int i = l; i < N / 2; i += kLevels) {
                        const float2 q = s_pair[e][i];
                        la += fminf(fabsf(q.x - (T[i] - T[i + N / 2])), q.y);
                    }
                    any = __any_sync(0xffffffffu, in && !(la > thr));
                    if (!any) break;
                }
                if (!any) continue;
            }
            float r[N];
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = s_w[e][i] > 0.0f ? s_obs[e][i] - T[i] : INF;
            bitonic_sort<N>(r);
            const int n = s_n[e], h = n / 2;
            float obj = 0.0f;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                /* lower half: i < h; upper half: n - h <= i < n (the middle one of
                 * an odd count drops out) */
                const float cf = i < h ? -1.0f : ((i >= n - h && i < n) ? 1.0f : 0.0f);
                obj = fmaf(cf, (i < n) ? r[i] : 0.0f, obj);
            }
            obj *= s_wv[e];
            const unsigned long long key = warp_min((in && n > 0) ? pack_key(obj, g) : ~0ull);
            if (lane == 0) {
                atomicMin(&s_best[e], key);
                atomicMin(&s_u[e], (unsigned)(key >> 32));
            }
        }
        __syncthreads();
        if (threadIdx.x < nb && s_best[threadIdx.x] != ~0ull) atomicMin(best + e0 + threadIdx.x, s_best[threadIdx.x]);
    }
}

/* One or two launches, as launch_l2_search. */
template <int N>
void launch_l1_search(int ngrd, int ldgrd, int ntf, const float *tables, int nev, const float *obs, const float *wts,
                      unsigned long long *best, cudaStream_t s)
{
    const long long ctas = (ngrd + (long long)kThreads - 1) / kThreads;
    const dim3 grid((unsigned)ctas, event_split(ctas, nev));
    if (ngrd < kBoundPoints) {
        l1_search_kernel<N, false><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, obs, wts, best);
        return;
    }
    const long long cs = ((ngrd + kSample - 1) / kSample + (long long)kThreads - 1) / kThreads;
    l1_search_kernel<N, false><<<dim3((unsigned)cs, event_split(cs, nev)), kThreads, 0, s>>>(
        ngrd, ldgrd, ntf, kSample, tables, nev, obs, wts, best);
    l1_search_kernel<N, true><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, obs, wts, best);
}

/* FP64 median and misfit at the chosen point from the FP64 picks
 * (insertion sort, one thread per event). */
__global__ void l1_at_opt_kernel(int ldgrd, int ntf, const float *__restrict__ tables, int nev,
                                 const double *__restrict__ obs, const double *__restrict__ wts,
                                 const unsigned long long *__restrict__ best, int *out_idx, double *out_t0,
                                 double *out_obj)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nev) return;
    const int g = (int)(best[e] & 0xffffffffu);
    double r[64];
    int n = 0;
    double wv = 0.0;
    for (int i = 0; i < ntf; ++i) {
        const double w = wts[(size_t)e * ntf + i];
        if (w > 0.0) {
            const double v = obs[(size_t)e * ntf + i] - (double)tables[(size_t)i * ldgrd + g];
            int j = n++;
            while (j > 0 && r[j - 1] > v) { r[j] = r[j - 1]; --j; }
            r[j] = v;
            wv = w;
        }
    }
    double t0 = 0.0, obj = 0.0;
    if (n > 0) {
        t0 = (n % 2) ? r[n / 2] : 0.5 * (r[n / 2 - 1] + r[n / 2]);
        for (int i = 0; i < n; ++i) obj += fabs(r[i] - t0);
        obj *= wv;
    }
    out_idx[e] = g;
    out_t0[e] = t0;
    out_obj[e] = obj;
}

__global__ void l1_init_kernel(int nev, unsigned long long *best)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < nev) best[e] = ~0ull;
}

} // namespace

extern "C" int fk_locate_l1_exact(int ngrd, int ldgrd, int ntf, const float *tables, int nev, const float *obs,
                                  const float *wts, const double *obs64, const double *wts64, int *out_idx,
                                  double *out_t0, double *out_obj, unsigned long long *scratch, cudaStream_t s)
{
    if (nev <= 0) return 0;
    if (ntf < 1 || ntf > kMaxTf) return (int)cudaErrorInvalidValue;
    l1_init_kernel<<<(nev + 255) / 256, 256, 0, s>>>(nev, scratch);
    if (ntf <= 16) launch_l1_search<16>(ngrd, ldgrd, ntf, tables, nev, obs, wts, scratch, s);
    else if (ntf <= 32) launch_l1_search<32>(ngrd, ldgrd, ntf, tables, nev, obs, wts, scratch, s);
    else launch_l1_search<64>(ngrd, ldgrd, ntf, tables, nev, obs, wts, scratch, s);
    l1_at_opt_kernel<<<(nev + 127) / 128, 128, 0, s>>>(ldgrd, ntf, tables, nev, obs64, wts64, scratch, out_idx,
                                                       out_t0, out_obj);
    return (int)cudaGetLastError();
}
