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
 * comes from a strided sample of the points.  Where FP32 ends (weights whose
 * squares or whose products with misfits leave its normal range) the bounds
 * allow for it or rule nothing out.
 *
 * Many events on a fine grid are bounded for 32 points at once first
 * (l2_block_kernel): over all picks the right-hand side is the square of a
 * seminorm of the weighted residuals that is zero for a common shift, so with
 * a block's point c, any tau(g) and d_i = max_g |T_i(g) - T_i(c) - tau(g)|
 *   sqrt(2 obj(g)) >= sqrt(s2 - s3^2 / sum w^2 at c) - sqrt(sum (w d)^2),
 * and a block is left out of an event's search if this exceeds the root of
 * twice its best objective.  tau is the mean over the tables of the
 * differences, which takes most of the times' common change out of d.
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
/* The relative errors above hold while nothing underflows or overflows: squares
 * of small terms lose at most 2^-149 each, with s3 / sum w^2 a difference of times
 * (up to 10^4) far below kSlackMin in all, if sum w^2 itself is far above 2^-149; a
 * sum w^2 outside [kSum2Min, kSum2Max] rules nothing out. */
constexpr float kSlackMin = 1e-36f, kSum2Min = 1e-36f, kSum2Max = 1e36f;

/* 1 / sum w^2; infinite, which makes the bound -infinity or a NaN, where it may not be used. */
__device__ __forceinline__ float bound_scale(float sum_w2)
{
    return sum_w2 >= kSum2Min && sum_w2 <= kSum2Max ? 1.0f / sum_w2 : __int_as_float(0x7f800000);
}

/* Searches the points p stride, p < np = ceil(ngrd / stride).  A warp owns 64
 * points, two per lane (32 apart, so every load is 4-byte and coalesced
 * whatever the tables' alignment) in packed FP32 arithmetic.  A CTA keeps its
 * tables while it runs over the events blockIdx.y, + gridDim.y, ... (in
 * chunks of kEvChunk).  BOUND: rule out by the bound first, level by level
 * (the sums carry on), while any of the warp's points survives.  The bound
 * costs 3 packed operations and one 16-byte shared-memory broadcast a pick.
 * The points are loaded, then evaluated, and the warps of the other CTAs of an
 * SM fill the gaps: 8, 4, 4 and 3 CTAs for 16, 32, 48 and 64 tables held.  One
 * event x 48 tables x 1.31e6 points 101 us a call with 48 tables held (4 CTAs),
 * 114 with 64 (3); 100 events x 14 x 542e3 183 us with 8 CTAs, 205 with 4; 40 x
 * 20 x 1.09e6 228 us with 4, 250 with 6. */
template <int NTF, bool BOUND>
__global__ void __launch_bounds__(kThreads, NTF == 64 ? 3 : NTF == 16 ? 8 : 4)
l2_search_kernel(int ngrd, int ldgrd, int ntf, int stride, const float *__restrict__ tables, int nev, int chunk,
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
    const int nchunk = (nev + chunk - 1) / chunk;
    for (int c = blockIdx.y; c < nchunk; c += gridDim.y) {
        const int e0 = c * chunk, nb = min(chunk, nev - e0);
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
            if (lane < kLevels) s_is2[e][lane] = bound_scale(a);
            if (lane == 0) {
                s_o2[e] = fmaf(kSlackO2, o2, kSlackMin);
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

/* kSlackD: d = max |T(g) - T(c) - tau| of the rounded differences falls short
 * of the exact one by 2 e d + 2 e |T(g) - T(c)| at most. */
constexpr float kSlackD = 1.0f / 2097152;  /* 2^-21 = 8 e */
constexpr int kBlkWarps = 8, kBlkThreads = 32 * kBlkWarps;
constexpr int kCtaBlk = 32;       /* blocks of 32 points of a CTA */
constexpr int kCtaPitch = kCtaBlk + 4;
constexpr int kGroup = 256;       /* events between two loads of the points' tables, at most */
constexpr int kChunk = 64;        /* events the blocks are tested for at a time */
constexpr int kBatch = 4;         /* events a warp evaluates at a time */
constexpr int kParts = 4;         /* the bound's subsets: 16 tables each, l, l + n, l + 2 n, ... of n parts */

/* Tables padded to whole steps of the unrolled loops, and the shared memory
 * for them: the blocks' centres and departures, and the chunk's picks or the
 * warps' points and events. */
__host__ __device__ inline int block_pad(int ntf) { return (ntf + 15) / 16 * 16; }
__host__ __device__ inline size_t block_smem(int ntf)
{
    const size_t per = 2 * kCtaPitch * sizeof(float),
                 chunk = (kChunk + 2) * sizeof(float2), points = kBlkWarps * (32 * sizeof(float) + kBatch * sizeof(float2));
    return block_pad(ntf) * (per + (chunk > points ? chunk : points));
}

/* An event's best objective so far; none yet: a NaN, which rules nothing out. */
__device__ __forceinline__ float best_so_far(const unsigned long long *best)
{
    return __uint_as_float(__ldcg(reinterpret_cast<const unsigned *>(best) + 1));
}

/* A block's tables into a warp's t[ntf][32]; a lane outside repeats the first point. */
__device__ __forceinline__ void block_points(float *t, const float *__restrict__ tables, int ldgrd, int ntf, int ngrd,
                                             long long g0, int lane)
{
    const float *src = tables + g0 + (g0 + lane < ngrd ? lane : 0);
    unsigned dst = (unsigned)__cvta_generic_to_shared(t + lane);
#pragma unroll 8
    for (int i = 0; i < ntf; ++i, src += ldgrd, dst += 32 * sizeof(float))
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void block_arrived()
{
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
}

/* The search of many events by blocks of points (see the file comment).  A CTA
 * owns 32 blocks.  First each block's T(c) and d go to shared memory.  Then,
 * for 64 events at a time, a thread bounds 4 blocks x 2 events (3 loads for
 * 20 packed multiply-adds a pick, bound by those).  Last the points of the
 * blocks left: a warp takes a block, brings its tables to shared memory and
 * evaluates four of its events at a time by the point bound, in parts, and
 * the objective where that does not rule them out.  All loops are short: a
 * version with the tables in registers and the loops over the picks unrolled
 * waited for instructions a third of its time (2.7 ms).  New best values go
 * to all CTAs at once.
 * 512 events x 64 tables x 2.46e6 points: 6.5 -> 2.1 ms a call, of which the
 * block bound takes 0.35, its preparation and the picks 0.4, the points 0.9
 * and the sample 0.2; 64 % of the issue slots are used.  CTAS to an SM: three
 * up to 32 tables (300 events x 30 x 1.1e6 points: 868 us against 940 with
 * two); above that the tables' shared memory (from 33 on 85 KB a CTA, its
 * static part and the reserve included, of 228) leaves room for two, and with
 * their registers 512 events x 33, 40, 48 tables x 266e3 points take 626, 662,
 * 713 us instead of 648, 682, 729. */
template <int CTAS>
__global__ void __launch_bounds__(kBlkThreads, CTAS)
l2_block_kernel(int ngrd, int ldgrd, int ntf, const float *__restrict__ tables, int nev, int group,
                const float *__restrict__ obs, const float *__restrict__ wts, const float *__restrict__ xnorm,
                unsigned long long *best)
{
    extern __shared__ __align__(16) unsigned char block_mem[];
    __shared__ float2 s_sum[kParts][kChunk];
    __shared__ float s_is2[kGroup][kParts], s_o2[kGroup], s_xn[kGroup];
    __shared__ unsigned s_live[kGroup / 32][kCtaBlk];    /* events a block is not ruled out for */
    __shared__ int s_next;
    static_assert(kBlkThreads == kParts * kChunk && kChunk == 8 * kBlkWarps && kCtaBlk == 32, "lanes are mapped to these");
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = block_pad(ntf), nl = nt / 16;
    float *const s_c = reinterpret_cast<float *>(block_mem), *const s_d = s_c + nt * kCtaPitch;   /* T at the centres, d */
    float2 *const s_pk = reinterpret_cast<float2 *>(s_d + nt * kCtaPitch);   /* [nt][kChunk + 2]: w, w o */
    float4 *const s_ev = reinterpret_cast<float4 *>(s_pk) + warp * (2 * nt);   /* [nt][2]: w, w o of four events */
    float *const s_t = reinterpret_cast<float *>(reinterpret_cast<float4 *>(s_pk) + kBlkWarps * 2 * nt) + warp * (32 * nt);
    const long long base = (long long)blockIdx.x * (kCtaBlk * 32);
    for (int i = ntf; i < nt; ++i) s_t[32 * i + lane] = 0.0f;
    for (int b = warp; b < kCtaBlk; b += kBlkWarps) { /* the blocks' centres and largest departures */
        const long long g0 = base + b * 32;
        if (g0 >= ngrd) break;
        const int cl = g0 + 16 < ngrd ? 16 : 0;
        __syncwarp();
        block_points(s_t, tables, ldgrd, ntf, ngrd, g0, lane);
        block_arrived();
        float sum = 0.0f;
#pragma unroll 8
        for (int i = 0; i < ntf; ++i) sum += s_t[32 * i + lane];
        const float tau = (sum - __shfl_sync(0xffffffffu, sum, cl)) / (float)ntf;
#pragma unroll 8
        for (int i = 0; i < nt; ++i) {
            const float c = s_t[32 * i + cl], a = s_t[32 * i + lane] - c;
            const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaf(kSlackD, fabsf(a), fabsf(a - tau))));
            if (lane == 0) {                              /* a NaN is the largest */
                s_c[i * kCtaPitch + b] = c;
                s_d[i * kCtaPitch + b] = __uint_as_float(m);
            }
        }
    }
    for (long long eg = (long long)blockIdx.y * group; eg < nev; eg += (long long)gridDim.y * group) {
        const int e0 = (int)eg, n = min(group, nev - e0);
        __syncthreads();
        if (tid == 0) s_next = 0;
        for (int e = tid; e < n; e += kBlkThreads) s_xn[e] = xnorm[e0 + e];
        s_live[warp][lane] = 0;
        for (int c0 = 0; c0 < n; c0 += kChunk) {
            const int nb = min(kChunk, n - c0);
            __syncthreads();
#pragma unroll
            for (int h = 0; h < kMaxTf; h += 32) {
                const int i = h + lane;
                if (h >= nt) break;
                float o[8], w[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int e = warp + kBlkWarps * k;
                    const bool on = e < nb && i < ntf;
                    o[k] = on ? obs[(size_t)(e0 + c0 + e) * ntf + i] : 0.0f;
                    w[k] = on ? wts[(size_t)(e0 + c0 + e) * ntf + i] : 0.0f;
                }
                if (i < nt) {
#pragma unroll
                    for (int k = 0; k < 8; ++k)                  /* a skipped pick has w = 0 */
                        s_pk[i * (kChunk + 2) + warp + kBlkWarps * k] =
                            w[k] > 0.0f ? make_float2(w[k], w[k] * o[k]) : make_float2(0.0f, 0.0f);
                }
            }
            __syncthreads();
            if (tid < kChunk * nl) {   /* 64 threads a part, one an event: sum w^2 and sum (w o)^2 */
                const int e = tid % kChunk, k = tid / kChunk;
                float a = 0.0f, o2 = 0.0f;
#pragma unroll 4
                for (int i = k; i < nt; i += nl) {
                    const float2 p = s_pk[i * (kChunk + 2) + e];
                    a = fmaf(p.x, p.x, a);
                    o2 = fmaf(p.y, p.y, o2);
                }
                s_sum[k][e] = make_float2(a, o2);
            }
            __syncthreads();
            if (tid < kChunk) {
                float a = 0.0f, o2 = 0.0f;
                for (int k = 0; k < nl; ++k) {
                    a += s_sum[k][tid].x;
                    o2 += s_sum[k][tid].y;
                    s_is2[c0 + tid][k] = bound_scale(a);
                }
                s_o2[c0 + tid] = fmaf(kSlackO2, o2, kSlackMin);
            }
            __syncthreads();
            /* the blocks: 4 of them (two packed pairs) and 2 events to a thread */
            const int b0 = 4 * (lane & 7), ev = 8 * warp + 2 * (lane >> 3);
            float2 s2[2][2], s3[2][2], d2[2][2];
#pragma unroll
            for (int k = 0; k < 4; ++k) s2[k / 2][k % 2] = s3[k / 2][k % 2] = d2[k / 2][k % 2] = dup(0.0f);
#pragma unroll 4
            for (int i = 0; i < nt; ++i) {
                const float4 c = *reinterpret_cast<const float4 *>(s_c + i * kCtaPitch + b0);
                const float4 d = *reinterpret_cast<const float4 *>(s_d + i * kCtaPitch + b0);
                const float4 pk = *reinterpret_cast<const float4 *>(s_pk + i * (kChunk + 2) + ev);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const float2 w = dup(k ? pk.z : pk.x), nw = dup(k ? -pk.z : -pk.x), wo = dup(k ? pk.w : pk.y);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const float2 p = __ffma2_rn(nw, j ? make_float2(c.z, c.w) : make_float2(c.x, c.y), wo);
                        const float2 r = __fmul2_rn(w, j ? make_float2(d.z, d.w) : make_float2(d.x, d.y));
                        s2[k][j] = __ffma2_rn(p, p, s2[k][j]);
                        s3[k][j] = __ffma2_rn(w, p, s3[k][j]);
                        d2[k][j] = __ffma2_rn(r, r, d2[k][j]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int e = c0 + ev + k;
                if (ev + k >= nb) break;
                const float is2 = s_is2[e][nl - 1], o2 = s_o2[e], u = best_so_far(best + e0 + e);
                const float root = sqrtf(fmaf(2.0f * u, 1.0f + kSlackObj, o2));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float a = j & 1 ? s2[k][j / 2].y : s2[k][j / 2].x, b = j & 1 ? s3[k][j / 2].y : s3[k][j / 2].x;
                    const float dd = j & 1 ? d2[k][j / 2].y : d2[k][j / 2].x;
                    const float lb = fmaf(-b * is2, b, fmaf(a, -kSlackS2, a)) - o2;
                    const float need = (root + fmaf(sqrtf(dd), 1.0f + kSlackS2, 1e-18f)) * (1.0f + kSlackO2);
                    if (base + (b0 + j) * 32 < ngrd && !(sqrtf(fmaxf(lb, 0.0f)) > need))
                        atomicOr(&s_live[e / 32][b0 + j], 1u << (e & 31));
                }
            }
        }
        __syncthreads();
        for (int i = ntf; i < nt; ++i) s_t[32 * i + lane] = 0.0f;
        /* the points of the blocks left: a block to a warp, four events at a time */
        for (;;) {
            int b = 0;
            if (lane == 0) b = atomicAdd(&s_next, 1);
            b = __shfl_sync(0xffffffffu, b, 0);
            if (b >= kCtaBlk) break;
            const unsigned mine = lane < kGroup / 32 ? s_live[lane][b] : 0;
            if (!__any_sync(0xffffffffu, mine)) continue;
            __syncwarp();
            block_points(s_t, tables, ldgrd, ntf, ngrd, base + b * 32, lane);
            const long long gl = base + b * 32 + lane;
            const bool in = gl < ngrd;
            const int g = in ? (int)gl : 0;
            int q = -1, ne[kBatch];                          /* the next events and their picks */
            unsigned left = 0;
            float po[kBatch][kMaxTf / 32] = {}, pw[kBatch][kMaxTf / 32] = {}, pu[kBatch];
            auto fetch = [&]() {
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    while (!left && q < kGroup / 32) left = __shfl_sync(0xffffffffu, mine, ++q);
                    ne[k] = left ? 32 * q + __ffs(left) - 1 : -1;
                    left &= left - 1;
                    pu[k] = ne[k] >= 0 ? best_so_far(best + e0 + ne[k]) : 0.0f;
#pragma unroll
                    for (int h = 0; h < kMaxTf / 32; ++h) {
                        if (h > 0 && 32 * h >= ntf) break;
                        const bool on = ne[k] >= 0 && 32 * h + lane < ntf;
                        po[k][h] = on ? __ldg(obs + (size_t)(e0 + ne[k]) * ntf + 32 * h + lane) : 0.0f;
                        pw[k][h] = on ? __ldg(wts + (size_t)(e0 + ne[k]) * ntf + 32 * h + lane) : 0.0f;
                    }
                }
            };
            fetch();
            block_arrived();
            while (ne[0] >= 0) {
                __syncwarp();
#pragma unroll
                for (int h = 0; h < kMaxTf / 32; ++h) {
                    if (h > 0 && 32 * h >= nt) break;
                    float4 v[2];
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const float w = pw[k][h] > 0.0f ? pw[k][h] : 0.0f, wo = pw[k][h] > 0.0f ? w * po[k][h] : 0.0f;
                        if (k & 1) { v[k / 2].z = w; v[k / 2].w = wo; } else { v[k / 2].x = w; v[k / 2].y = wo; }
                    }
                    if (32 * h + lane < nt) {
                        s_ev[2 * (32 * h + lane)] = v[0];
                        s_ev[2 * (32 * h + lane) + 1] = v[1];
                    }
                }
                __syncwarp();
                int e[kBatch];
                bool x[kBatch];
                float thr[kBatch], s2[kBatch], s3[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    x[k] = ne[k] >= 0;
                    e[k] = x[k] ? ne[k] : ne[0];
                    thr[k] = fmaf(2.0f * pu[k], 1.0f + kSlackObj, s_o2[e[k]]);
                    s2[k] = s3[k] = 0.0f;
                }
                fetch();
#pragma unroll 1
                for (int l = 0; l < nl; ++l) {
                    const float *pt = s_t + 32 * l + lane;
                    const float4 *pe = s_ev + 2 * l;
#pragma unroll
                    for (int j = 0; j < 16; ++j, pt += 32 * nl, pe += 2 * nl) {
                        const float t = *pt;
                        const float4 pa = pe[0], pb = pe[1];
                        const float w[kBatch] = {pa.x, pa.z, pb.x, pb.z}, wo[kBatch] = {pa.y, pa.w, pb.y, pb.w};
#pragma unroll
                        for (int k = 0; k < kBatch; ++k) {
                            const float p = fmaf(-w[k], t, wo[k]);
                            s2[k] = fmaf(p, p, s2[k]);
                            s3[k] = fmaf(w[k], p, s3[k]);
                        }
                    }
                    bool any = false;
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        const float lb = fmaf(-s3[k] * s_is2[e[k]][l], s3[k], fmaf(s2[k], -kSlackS2, s2[k]));
                        x[k] = __any_sync(0xffffffffu, in && x[k] && !(lb > thr[k]));
                        any |= x[k];
                    }
                    if (!any) break;
                }
#pragma unroll 1
                for (int k = 0; k < kBatch; ++k) {
                    const bool on = k == 0 ? x[0] : k == 1 ? x[1] : k == 2 ? x[2] : x[3];
                    if (!on) continue;
                    const int ek = k == 0 ? e[0] : k == 1 ? e[1] : k == 2 ? e[2] : e[3];
                    float o[kMaxTf / 32], w[kMaxTf / 32];
#pragma unroll
                    for (int h = 0; h < kMaxTf / 32; ++h) {
                        const bool use = 32 * h + lane < ntf;
                        o[h] = use ? __ldg(obs + (size_t)(e0 + ek) * ntf + 32 * h + lane) : 0.0f;
                        w[h] = use ? __ldg(wts + (size_t)(e0 + ek) * ntf + 32 * h + lane) : 0.0f;
                    }
                    const float xn = s_xn[ek];
                    float t0 = 0.0f, obj = 0.0f;             /* as l2_search_kernel's, in its order */
#pragma unroll 4
                    for (int i = 0; i < ntf; ++i) {
                        const float oi = __shfl_sync(0xffffffffu, i < 32 ? o[0] : o[1], i & 31);
                        const float wi = __shfl_sync(0xffffffffu, i < 32 ? w[0] : w[1], i & 31);
                        const float t = __fadd_rn(t0, __fmul_rn(wi, __fmul_rn(xn, __fsub_rn(oi, s_t[32 * i + lane]))));
                        t0 = wi > 0.0f ? t : t0;
                    }
#pragma unroll 4
                    for (int i = 0; i < ntf; ++i) {
                        const float oi = __shfl_sync(0xffffffffu, i < 32 ? o[0] : o[1], i & 31);
                        const float wi = __shfl_sync(0xffffffffu, i < 32 ? w[0] : w[1], i & 31);
                        const float res = __fmul_rn(__fmul_rn(0.70710677f, wi), __fsub_rn(oi, __fadd_rn(s_t[32 * i + lane], t0)));
                        obj = wi > 0.0f ? __fadd_rn(obj, __fmul_rn(res, res)) : obj;
                    }
                    const unsigned long long key = warp_min(in ? pack_key(obj, g) : ~0ull);
                    if (lane == 0) atomicMin(best + e0 + ek, key);
                }
            }
        }
    }
}

/* Sum of kMaxTf values in shared memory, in order (16-byte loads a few ahead of
 * the chain of additions). */
__device__ __forceinline__ float ordered_sum(const float *v, int n)
{
    float s = 0.0f;
#pragma unroll 4
    for (int i = 0; i < n; i += 4) {
        const float4 q = *reinterpret_cast<const float4 *>(v + i);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, q.x), q.y), q.z), q.w);
    }
    return s;
}

/* t0 and obj at the optimum, same arithmetic: a warp per event forms its terms,
 * two a lane, and adds them in order; a skipped pick's is +0, which leaves a
 * sum that started at +0 as it is.  With one lane forming and adding all terms
 * the kernel took 7.5 us for one event, so 5.6 (one event x 45 tables x 542e3
 * points 73.7 -> 67.4 us a call, the weights' sum below included). */
__global__ void __launch_bounds__(128)
l2_at_opt_kernel(int ldgrd, int ntf, const float *__restrict__ tables, int nev, const float *__restrict__ obs,
                 const float *__restrict__ wts, const float *__restrict__ xnorm,
                 const unsigned long long *__restrict__ best, int *out_idx, float *out_t0, float *out_obj)
{
    __shared__ __align__(16) float s_term[4][2][kMaxTf];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.x * 4 + warp;
    if (e >= nev) return;
    const int g = (int)(best[e] & 0xffffffffu);
    const float xn = xnorm[e];
    float o[kMaxTf / 32], w[kMaxTf / 32], T[kMaxTf / 32];
#pragma unroll
    for (int h = 0; h < kMaxTf / 32; ++h) {
        const int i = 32 * h + lane;
        const bool in = i < ntf;
        o[h] = in ? obs[(size_t)e * ntf + i] : 0.0f;
        w[h] = in ? wts[(size_t)e * ntf + i] : 0.0f;
        T[h] = in ? tables[(size_t)i * ldgrd + g] : 0.0f;
        s_term[warp][0][i] = w[h] > 0.0f ? __fmul_rn(w[h], __fmul_rn(xn, __fsub_rn(o[h], T[h]))) : 0.0f;
    }
    __syncwarp();
    const int n4 = (ntf + 3) / 4 * 4;
    const float t0 = ordered_sum(s_term[warp][0], n4);
#pragma unroll
    for (int h = 0; h < kMaxTf / 32; ++h) {
        const float res = __fmul_rn(__fmul_rn(0.70710677f, w[h]), __fsub_rn(o[h], __fadd_rn(T[h], t0)));
        s_term[warp][1][32 * h + lane] = w[h] > 0.0f ? __fmul_rn(res, res) : 0.0f;
    }
    __syncwarp();
    const float obj = ordered_sum(s_term[warp][1], n4);
    if (lane == 0) {
        out_idx[e] = g;
        out_t0[e] = t0;
        out_obj[e] = obj;
    }
}

/* 1 / SUM over the padded weight row, in order; a warp per event. */
__global__ void __launch_bounds__(128) xnorm_kernel(int nev, int ntf, const float *__restrict__ wts, float *xnorm,
                                                    unsigned long long *best)
{
    __shared__ __align__(16) float s_w[4][kMaxTf];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int e = blockIdx.x * 4 + warp;
    if (e >= nev) return;
    for (int i = lane; i < kMaxTf; i += 32) s_w[warp][i] = i < ntf ? wts[(size_t)e * ntf + i] : 0.0f;
    __syncwarp();
    if (lane == 0) {
        xnorm[e] = __fdiv_rn(1.0f, ordered_sum(s_w[warp], (ntf + 3) / 4 * 4));
        best[e] = ~0ull;
    }
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
/* Blocks of points pay from about 200 events (their centres and departures
 * cost as much as some 100 events' point bounds) and on fine grids, where the
 * times change little within 32 points; above 48 tables, where the blocks'
 * centres and the warps' points are dearest, the grid has to be larger.  By
 * points / by blocks, us: 192 events x 269e3 points x 14, 30, 60 tables
 * 198 / 183, 249 / 243, 387 / 412; 256 events x 266e3 x 33, 40, 48 491 / 469,
 * 504 / 502, 532 / 531 (192 events 391 / 402, 403 / 428, 432 / 455), x 410e3
 * 600 / 441, 608 / 471, 646 / 505;
 * x 542e3 x 60 673 / 668; x 1.09e6 x 60 1311 / 1141; 60 events x 600e3 x 20
 * 183 / 207; 300 events x 99e3 x 32 210 / 250; 500 events x 256e3 x 20
 * 496 / 382. */
constexpr int kBlockEvents = 192;
inline int block_points(int ntf) { return ntf <= 48 ? 1 << 18 : 1 << 19; }

/* Grid of the point kernels: their CTAs over the points, and over the events
 * when those leave the chip idle (148 SMs, 3 CTAs each, a few waves); chunks of
 * fewer events when that still does, as in the sample of a small grid. */
inline dim3 point_grid(long long ctas, int nev, int *chunk)
{
    *chunk = kEvChunk;
    while (*chunk > 1 && ctas * ((nev + *chunk - 1) / *chunk) < 148 * 3) *chunk /= 2;
    const int nchunk = (nev + *chunk - 1) / *chunk;
    const long long y = (148 * 3 * 4 + ctas - 1) / ctas;
    return dim3((unsigned)ctas, (unsigned)(y < 1 ? 1 : y > nchunk ? nchunk : y));
}

/* Grid of the block kernels: the blocks, and events in groups, smaller ones
 * when the points alone leave the chip idle. */
inline dim3 block_grid(int ngrd, int nev, int *group)
{
    const long long cb = (ngrd + 32ll * kCtaBlk - 1) / (32 * kCtaBlk);
    *group = kGroup;
    while (*group > kChunk / 2 && cb * ((nev + *group - 1) / *group) < 148 * 2 * 4) *group /= 2;
    const long long y = (148 * 2 * 4 + cb - 1) / cb, ng = (nev + *group - 1) / *group;
    return dim3((unsigned)cb, (unsigned)(y < 1 ? 1 : y > ng ? ng : y));
}

template <int NTF>
cudaError_t launch_l2_search(int ngrd, int ldgrd, int ntf, const float *tables, int nev, const float *obs, const float *wts,
                             const float *xn, unsigned long long *best, cudaStream_t s)
{
    const int per = kThreads / 32 * 64;
    const long long ctas = (ngrd + (long long)per - 1) / per;
    int chunk;
    const dim3 grid = point_grid(ctas, nev, &chunk);
    if (nev < kBoundEvents || ngrd < kBoundPoints) {
        l2_search_kernel<NTF, false><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, chunk, obs, wts, xn, best);
        return cudaSuccess;
    }
    const long long cs = ((ngrd + (long long)kSample - 1) / kSample + (long long)per - 1) / per;
    int schunk;
    const dim3 sgrid = point_grid(cs, nev, &schunk);
    l2_search_kernel<NTF, false><<<sgrid, kThreads, 0, s>>>(
        ngrd, ldgrd, ntf, kSample, tables, nev, schunk, obs, wts, xn, best);
    if (nev < kBlockEvents || ngrd < block_points(ntf)) {
        l2_search_kernel<NTF, true><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, chunk, obs, wts, xn, best);
        return cudaSuccess;
    }
    int group;
    const dim3 gb = block_grid(ngrd, nev, &group);
    const size_t smem = block_smem(ntf);
    auto *kernel = ntf <= 32 ? l2_block_kernel<3> : l2_block_kernel<2>;
    /* the limit for the widest tables it serves: calls of other threads may set it too */
    const cudaError_t ea = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                (int)block_smem(ntf <= 32 ? 32 : kMaxTf));
    if (ea != cudaSuccess) return ea;
    kernel<<<gb, kBlkThreads, smem, s>>>(
        ngrd, ldgrd, ntf, tables, nev, group, obs, wts, xn, best);
    return cudaSuccess;
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
    xnorm_kernel<<<(nev + 3) / 4, 128, 0, s>>>(nev, ntf, wts, xn, best);
    auto *search = ntf <= 16   ? launch_l2_search<16>
                   : ntf <= 32 ? launch_l2_search<32>
                   : ntf <= 48 ? launch_l2_search<48>
                               : launch_l2_search<64>;
    const cudaError_t e = search(ngrd, ldgrd, ntf, tables, nev, obs, wts, xn, best, s);
    if (e != cudaSuccess) return (int)e;
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
/* out first by a bound on the misfit (l1_search_kernel), of many events on */
/* large grids 32 at a time (l1_block_kernel).  The argmin is               */
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

/* Misfit per unit weight of n residuals (the others +inf); sorts them. */
template <int N>
__device__ __forceinline__ float l1_sorted_misfit(float (&r)[N], int n)
{
    bitonic_sort<N>(r);
    const int h = n / 2;
    float obj = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        /* lower half: i < h; upper half: n - h <= i < n (the middle one of
         * an odd count drops out) */
        const float cf = i < h ? -1.0f : ((i >= n - h && i < n) ? 1.0f : 0.0f);
        obj = fmaf(cf, (i < n) ? r[i] : 0.0f, obj);
    }
    return obj;
}

/* Rounding allowance of the L1 bound: with e = 2^-24 the ranking misfit is
 * computed to (N + 1) e sum (|o| + |T|) and the pairs' sum to (N / 2 + 4) e of
 * the same, N <= 64 (times the event's weight). */
constexpr float kSlackL1 = 1.0f / 131072;   /* 2^-17 = 128 e */

/* An event's share of what kSlackL1 applies to, so = sum |o|.  The ranked product
 * of misfit and weight is rounded to 2^-149 at least, which moves a misfit by
 * 2^-150 / w: less than kSlackL1 1e-15 for weights down to 1e-25; below, nothing
 * is ruled out. */
__device__ __forceinline__ float l1_slack_obs(float so, float w)
{
    return w >= 1e-25f ? so + 1e-15f : __int_as_float(0x7f800000);
}

/* Searches the points p stride; a warp owns 32 points, one a lane, and runs
 * over the events as l2_search_kernel does.  BOUND: for any t0 two picks
 * give |r_i - t0| + |r_j - t0| >= |r_i - r_j|, so the sum over disjoint pairs
 * (2 i, 2 i + 1) bounds the misfit from below at four operations a pair,
 * against the sorting network's 672 compare-exchanges for 64 picks; the
 * pairs come in kLevels levels, and a point is sorted only if all of them
 * stay below the event's best misfit so far.  A pair with a skipped pick
 * counts zero (its cap).  128 events x 64 tables x 2.46e6 points: 3.3 ms
 * (3.7 and 3.4 ms with every 64th and 1024th point in the sample) against
 * 38.6 ms with every point sorted. */
template <int N, bool BOUND>
__global__ void __launch_bounds__(kThreads, 3)
l1_search_kernel(int ngrd, int ldgrd, int ntf, int stride, const float *__restrict__ tables, int nev, int chunk,
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
    const int nchunk = (nev + chunk - 1) / chunk;
    for (int c = blockIdx.y; c < nchunk; c += gridDim.y) {
        const int e0 = c * chunk, nb = min(chunk, nev - e0);
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
                    s_pair[e][i] = make_float2(s_obs[e][2 * i] - s_obs[e][2 * i + 1],
                                               s_w[e][2 * i] > 0.0f && s_w[e][2 * i + 1] > 0.0f ? INF : 0.0f);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                n += __shfl_xor_sync(0xffffffffu, n, o);
                wv = fmaxf(wv, __shfl_xor_sync(0xffffffffu, wv, o));   /* one weight per event */
                so += __shfl_xor_sync(0xffffffffu, so, o);
            }
            if (lane == 0) {
                s_n[e] = n;
                s_wv[e] = wv;
                s_o[e] = l1_slack_obs(so, wv);
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
                        la += fminf(fabsf(q.x - (T[2 * i] - T[2 * i + 1])), q.y);
                    }
                    any = __any_sync(0xffffffffu, in && !(la > thr));
                    if (!any) break;
                }
                if (!any) continue;
            }
            float r[N];
#pragma unroll
            for (int i = 0; i < N; ++i) r[i] = s_w[e][i] > 0.0f ? s_obs[e][i] - T[i] : INF;
            const int n = s_n[e];
            const float obj = l1_sorted_misfit<N>(r, n) * s_wv[e];
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

/* Shared memory of l1_block_kernel: a block's pairs at its centre and their
 * departures, and the chunk's pairs or the warps' points, events and picks. */
__host__ __device__ inline int l1_pairs_pad(int ntf) { return (ntf / 2 + 7) / 8 * 8; }
inline size_t l1_block_smem(int ntf)
{
    const size_t np = l1_pairs_pad(ntf), per = 2 * kCtaPitch * np, chunk = (kChunk + 2) * np,
                 points = kBlkWarps * (32 * ntf + kBatch * np + 2 * kMaxTf);
    return sizeof(float) * (per + (chunk > points ? chunk : points));
}

/* The search of many events by blocks of 32 points, as l2_block_kernel.  The
 * bound's pairs are picks i and i + ntf / 2: with a block's centre c and
 * d = max_g |(T_i - T_j)(g) - (T_i - T_j)(c)| a pair gives at least
 * max(0, |o_i - o_j - (T_i - T_j)(c)| - d) anywhere in the block.  A pair with
 * a skipped pick is a NaN, which the maximum turns into zero.  The rounding
 * errors of the bound, (N / 2 + 6) e of sum |o|, sum |T| and the departures,
 * and of the ranking misfit stay below twice kSlackL1 (|o| + |T|).
 * 128 events x 64 tables x 2.46e6 points: 3.3 -> 1.28 ms a call. */
template <int N>
__global__ void __launch_bounds__(kBlkThreads, N == 64 ? 2 : 3)
l1_block_kernel(int ngrd, int ldgrd, int ntf, const float *__restrict__ tables, int nev, int group,
                const float *__restrict__ obs, const float *__restrict__ wts, unsigned long long *best)
{
    extern __shared__ __align__(16) unsigned char block_mem[];
    __shared__ float s_wv[kGroup], s_o[kGroup], s_far[kCtaBlk];   /* weight, sum |o|; largest sum |T| */
    __shared__ int s_n[kGroup];
    __shared__ unsigned s_live[kGroup / 32][kCtaBlk];
    __shared__ int s_next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = ntf / 2, np = l1_pairs_pad(ntf);
    const float INF = __int_as_float(0x7f800000), NONE = __int_as_float(0x7fffffff);
    float *const s_c = reinterpret_cast<float *>(block_mem), *const s_d = s_c + np * kCtaPitch;
    float *const s_q = s_d + np * kCtaPitch;                        /* [np][kChunk + 2]: o_i - o_j */
    float4 *const s_ev = reinterpret_cast<float4 *>(s_q) + warp * np;   /* of four events */
    float2 *const s_ow = reinterpret_cast<float2 *>(reinterpret_cast<float4 *>(s_q) + kBlkWarps * np) + warp * kMaxTf;
    float *const s_t = s_q + kBlkWarps * (kBatch * np + 2 * kMaxTf) + warp * (32 * ntf);
    const long long base = (long long)blockIdx.x * (kCtaBlk * 32);
    for (int b = warp; b < kCtaBlk; b += kBlkWarps) {
        const long long g0 = base + b * 32;
        if (g0 >= ngrd) break;
        const int cl = g0 + 16 < ngrd ? 16 : 0;
        __syncwarp();
        block_points(s_t, tables, ldgrd, ntf, ngrd, g0, lane);
        block_arrived();
        float sum = 0.0f;
#pragma unroll 8
        for (int i = 0; i < ntf; ++i) sum += fabsf(s_t[32 * i + lane]);
        const unsigned far = __reduce_max_sync(0xffffffffu, __float_as_uint(sum));
        if (lane == 0) s_far[b] = __uint_as_float(far);
#pragma unroll 4
        for (int i = 0; i < np; ++i) {
            float c = 0.0f;
            unsigned m = 0;
            if (i < half) {
                const float t = s_t[32 * i + lane] - s_t[32 * (i + half) + lane];
                c = __shfl_sync(0xffffffffu, t, cl);
                m = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(t - c)));   /* a NaN is the largest */
            }
            if (lane == 0) {
                s_c[i * kCtaPitch + b] = c;
                s_d[i * kCtaPitch + b] = __uint_as_float(m);
            }
        }
    }
    for (long long eg = (long long)blockIdx.y * group; eg < nev; eg += (long long)gridDim.y * group) {
        const int e0 = (int)eg, n = min(group, nev - e0);
        __syncthreads();
        if (tid == 0) s_next = 0;
        s_live[warp][lane] = 0;
        for (int c0 = 0; c0 < n; c0 += kChunk) {
            const int nb = min(kChunk, n - c0);
            __syncthreads();
#pragma unroll 4
            for (int k = 0; k < kChunk / kBlkWarps; ++k) {       /* a warp an event, a lane a pair */
                const int e = warp + kBlkWarps * k;
                const float *po = obs + (size_t)(e0 + c0 + e) * ntf, *pw = wts + (size_t)(e0 + c0 + e) * ntf;
                const bool a = e < nb && lane < half, last = e < nb && lane == 0 && (ntf & 1);
                const float oi = a ? po[lane] : 0.0f, wi = a ? pw[lane] : 0.0f;
                const float oj = a ? po[lane + half] : 0.0f, wj = a ? pw[lane + half] : 0.0f;
                const float ol = last ? po[ntf - 1] : 0.0f, wl = last ? pw[ntf - 1] : 0.0f;
                const bool ui = wi > 0.0f, uj = wj > 0.0f, ul = wl > 0.0f;
                const int cnt = __popc(__ballot_sync(0xffffffffu, ui)) + __popc(__ballot_sync(0xffffffffu, uj)) +
                                __popc(__ballot_sync(0xffffffffu, ul));
                const unsigned wv = __reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(fmaxf(ui ? wi : 0.0f, uj ? wj : 0.0f),
                                                                                        ul ? wl : 0.0f)));
                float so = (ui ? fabsf(oi) : 0.0f) + (uj ? fabsf(oj) : 0.0f) + (ul ? fabsf(ol) : 0.0f);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) so += __shfl_xor_sync(0xffffffffu, so, o);
                if (lane < np) s_q[lane * (kChunk + 2) + e] = ui && uj ? oi - oj : NONE;
                if (lane == 0) {
                    s_n[c0 + e] = cnt;
                    s_wv[c0 + e] = __uint_as_float(wv);       /* one weight per event */
                    s_o[c0 + e] = l1_slack_obs(so, __uint_as_float(wv));
                }
            }
            __syncthreads();
            const int b0 = 4 * (lane & 7), ev = 8 * warp + 2 * (lane >> 3);
            float la[2][4] = {};
#pragma unroll 8
            for (int i = 0; i < np; ++i) {
                const float4 c4 = *reinterpret_cast<const float4 *>(s_c + i * kCtaPitch + b0);
                const float4 d4 = *reinterpret_cast<const float4 *>(s_d + i * kCtaPitch + b0);
                const float2 q = *reinterpret_cast<const float2 *>(s_q + i * (kChunk + 2) + ev);
                const float c[4] = {c4.x, c4.y, c4.z, c4.w}, d[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    la[0][j] += fmaxf(fabsf(q.x - c[j]) - d[j], 0.0f);
                    la[1][j] += fmaxf(fabsf(q.y - c[j]) - d[j], 0.0f);
                }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int e = c0 + ev + k;
                if (ev + k >= nb) break;
                const float u = best_so_far(best + e0 + e), most = u / s_wv[e] * (1.0f + 1.0f / 1048576);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    /* a misfit of -0 or rounded below zero orders after all others (its key is unsigned) */
                    const float thr = signbit(u) ? INF : fmaf(2.0f * kSlackL1, s_far[b0 + j] + s_o[e], most);
                    if (base + (b0 + j) * 32 < ngrd && !(la[k][j] > thr)) atomicOr(&s_live[e / 32][b0 + j], 1u << (e & 31));
                }
            }
        }
        __syncthreads();
        for (;;) {
            int b = 0;
            if (lane == 0) b = atomicAdd(&s_next, 1);
            b = __shfl_sync(0xffffffffu, b, 0);
            if (b >= kCtaBlk) break;
            const unsigned mine = lane < kGroup / 32 ? s_live[lane][b] : 0;
            if (!__any_sync(0xffffffffu, mine)) continue;
            __syncwarp();
            block_points(s_t, tables, ldgrd, ntf, ngrd, base + b * 32, lane);
            const long long gl = base + b * 32 + lane;
            const bool in = gl < ngrd;
            const int g = in ? (int)gl : 0;
            int q = -1, ne[kBatch];                              /* the next events and their pairs */
            unsigned left = 0;
            float poi[kBatch], poj[kBatch], pwi[kBatch], pwj[kBatch], pu[kBatch];
            auto fetch = [&]() {
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    while (!left && q < kGroup / 32) left = __shfl_sync(0xffffffffu, mine, ++q);
                    ne[k] = left ? 32 * q + __ffs(left) - 1 : -1;
                    left &= left - 1;
                    pu[k] = ne[k] >= 0 ? best_so_far(best + e0 + ne[k]) : 0.0f;
                    const bool on = ne[k] >= 0 && lane < half;
                    const size_t at = (size_t)(e0 + (on ? ne[k] : 0)) * ntf + (on ? lane : 0);
                    poi[k] = __ldg(obs + at);
                    poj[k] = __ldg(obs + at + half);
                    pwi[k] = on ? __ldg(wts + at) : 0.0f;
                    pwj[k] = __ldg(wts + at + half);
                }
            };
            fetch();
            block_arrived();
            float sumT = 0.0f;
#pragma unroll 8
            for (int i = 0; i < ntf; ++i) sumT += fabsf(s_t[32 * i + lane]);
            while (ne[0] >= 0) {
                __syncwarp();
                float v[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) v[k] = pwi[k] > 0.0f && pwj[k] > 0.0f ? poi[k] - poj[k] : NONE;
                if (lane < np) s_ev[lane] = make_float4(v[0], v[1], v[2], v[3]);
                __syncwarp();
                int e[kBatch];
                bool x[kBatch];
                float thr[kBatch], la[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    x[k] = ne[k] >= 0;
                    e[k] = x[k] ? ne[k] : ne[0];
                    thr[k] = signbit(pu[k]) ? INF
                                            : fmaf(pu[k] / s_wv[e[k]], 1.0f + 1.0f / 1048576, kSlackL1 * (sumT + s_o[e[k]]));
                    la[k] = 0.0f;
                }
                fetch();
#pragma unroll 1
                for (int l = 0; l < np; l += 8) {
#pragma unroll
                    for (int i = l; i < l + 8; ++i) {
                        if (i >= half) break;
                        const float t = s_t[32 * i + lane] - s_t[32 * (i + half) + lane];
                        const float4 v = s_ev[i];
                        la[0] += fmaxf(fabsf(v.x - t), 0.0f);
                        la[1] += fmaxf(fabsf(v.y - t), 0.0f);
                        la[2] += fmaxf(fabsf(v.z - t), 0.0f);
                        la[3] += fmaxf(fabsf(v.w - t), 0.0f);
                    }
                    bool any = false;
#pragma unroll
                    for (int k = 0; k < kBatch; ++k) {
                        x[k] = __any_sync(0xffffffffu, in && x[k] && !(la[k] > thr[k]));
                        any |= x[k];
                    }
                    if (!any) break;
                }
#pragma unroll 1
                for (int k = 0; k < kBatch; ++k) {
                    if (!(k == 0 ? x[0] : k == 1 ? x[1] : k == 2 ? x[2] : x[3])) continue;
                    const int ek = k == 0 ? e[0] : k == 1 ? e[1] : k == 2 ? e[2] : e[3];
                    __syncwarp();
                    for (int i = lane; i < ntf; i += 32)
                        s_ow[i] = make_float2(__ldg(obs + (size_t)(e0 + ek) * ntf + i), __ldg(wts + (size_t)(e0 + ek) * ntf + i));
                    __syncwarp();
                    float r[N];
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        r[i] = INF;
                        if (i < ntf) {
                            const float2 ow = s_ow[i];
                            if (ow.y > 0.0f) r[i] = ow.x - s_t[32 * i + lane];
                        }
                    }
                    const int m = s_n[ek];
                    const float obj = l1_sorted_misfit<N>(r, m) * s_wv[ek];
                    const unsigned long long key = warp_min((in && m > 0) ? pack_key(obj, g) : ~0ull);
                    if (lane == 0) atomicMin(best + e0 + ek, key);
                }
            }
        }
    }
}

/* Where blocks pay, as for L2; the point bound is dear here, so earlier.  By
 * points / by blocks, us: 100 events x 99e3 points x 20 tables 206 / 155, 30
 * events x 144e3 x 20 128 / 128, 10 x 99e3 x 20 81 / 99; above 32 tables (64
 * residuals to sort, two CTAs to an SM) 100 x 144e3 x 60 430 / 468, 20 x 541e3
 * x 60 336 / 348, 64 x 541e3 x 60 679 / 542. */
inline int l1_block_events(int ntf) { return ntf <= 32 ? 32 : 64; }
inline int l1_block_points(int ntf) { return ntf <= 32 ? 1 << 16 : 1 << 18; }

/* One or two launches, as launch_l2_search. */
template <int N>
cudaError_t launch_l1_search(int ngrd, int ldgrd, int ntf, const float *tables, int nev, const float *obs, const float *wts,
                             unsigned long long *best, cudaStream_t s)
{
    const long long ctas = (ngrd + (long long)kThreads - 1) / kThreads;
    int chunk;
    const dim3 grid = point_grid(ctas, nev, &chunk);
    if (ngrd < kBoundPoints) {
        l1_search_kernel<N, false><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, chunk, obs, wts, best);
        return cudaSuccess;
    }
    const long long cs = ((ngrd + (long long)kSample - 1) / kSample + (long long)kThreads - 1) / kThreads;
    int schunk;
    const dim3 sgrid = point_grid(cs, nev, &schunk);
    l1_search_kernel<N, false><<<sgrid, kThreads, 0, s>>>(
        ngrd, ldgrd, ntf, kSample, tables, nev, schunk, obs, wts, best);
    if (nev < l1_block_events(ntf) || ngrd < l1_block_points(ntf)) {
        l1_search_kernel<N, true><<<grid, kThreads, 0, s>>>(ngrd, ldgrd, ntf, 1, tables, nev, chunk, obs, wts, best);
        return cudaSuccess;
    }
    int group;
    const dim3 gb = block_grid(ngrd, nev, &group);
    const size_t smem = l1_block_smem(ntf);
    const cudaError_t ea =
        cudaFuncSetAttribute(l1_block_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)l1_block_smem(N));
    if (ea != cudaSuccess) return ea;
    l1_block_kernel<N><<<gb, kBlkThreads, smem, s>>>(ngrd, ldgrd, ntf, tables, nev, group, obs, wts, best);
    return cudaSuccess;
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
    /* weights that vanish in FP32 leave no key: every ranked misfit is zero, the first point the optimum */
    const int g = best[e] == ~0ull ? 0 : (int)(best[e] & 0xffffffffu);
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
    auto *search = ntf <= 16 ? launch_l1_search<16> : ntf <= 32 ? launch_l1_search<32> : launch_l1_search<64>;
    const cudaError_t e = search(ngrd, ldgrd, ntf, tables, nev, obs, wts, scratch, s);
    if (e != cudaSuccess) return (int)e;
    l1_at_opt_kernel<<<(nev + 127) / 128, 128, 0, s>>>(ldgrd, ntf, tables, nev, obs64, wts64, scratch, out_idx,
                                                       out_t0, out_obj);
    return (int)cudaGetLastError();
}
