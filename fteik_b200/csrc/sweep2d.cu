/*
 * sweep2d.cu -- the reference's 2D level-set solve (solver2D.F90:782-978,
 * node updates localSolver.F90:123-289) and its natural-order twin
 * solveSourceFSM (solver2D.F90:1042-1280), in FP64.
 *
 * Grids up to 512 columns take the diagonal walk (second half of the file);
 * wider ones, solves to convergence, and those for whose scratch the device has
 * no memory left, the walk in place:
 *
 * One CTA owns one (grid, source).  Thread t owns the logical x columns
 * b NT + t (b = 0, 1, ...: column blocks of NT <= 512 threads) and walks
 * their z positions, block after block, thread t one step behind thread t-1,
 * so tv is the thread's previous result, te the previous result of thread
 * t-1 (warp shuffle, the two-slot hand-off between warps, or for thread 0 of
 * block b > 0 the last thread's result of block b-1 through a ring indexed
 * by z, Zb >= NT steps old) and tev the thread's previous te.  Both reference
 * schedules are topological orders of the same dependency graph, so LSM and
 * FSM give identical fields here (the FSM's initialisation box clamp is
 * applied to both).  Compiled without multiply-add contraction.
 */
#include <cuda_runtime.h>
#include "fteik_dev.h"
#include "fp64.cuh"

namespace {

constexpr int kMaxWarps = 16;
constexpr int kMaxThreads = kMaxWarps * 32;   /* 512: 128 registers per thread, no spills */

struct Mesh2 {
    double dz, dx, dzi, dxi, dz2i, dx2i, dz2i_dx2i, dz2i_p_dx2i, dz2i_p_dx2i_inv;
};

struct Src2 {
    int zsi, xsi;
    double zsa, xsa, szero, eps;
};

__device__ __forceinline__ double dmin(double a, double b) { return (b < a) ? b : a; }

/* localSolver.F90:36-50 */
__device__ __forceinline__ double tana2(const Src2 &q, const Mesh2 &c, int i, int j)
{
    double dz_ = ((double)i - q.zsa) * c.dz;
    double dx_ = ((double)j - q.xsa) * c.dx;
    return q.szero * hypot(dx_, dz_);
}

/* localSolver.F90:123-158 */
__device__ __forceinline__ double noinit2(const Mesh2 &c, double tv, double te,
                                          double tev, double s1, double s2, double s3)
{
    double temtv = te - tv;
    double t12min = dmin(tv + c.dz * s1, te + c.dx * s2);
    double t1_2d = FK_HUGE;
    if (temtv < c.dz * s3 && -temtv < c.dx * s3) {
        double ta = tev + temtv, tb = tev - temtv, tab = ta - tb;
        t1_2d = ((tb * c.dz2i + ta * c.dx2i) +
                 sqrt((4.0 * (s3 * s3)) * c.dz2i_p_dx2i - c.dz2i_dx2i * (tab * tab))) *
                c.dz2i_p_dx2i_inv;
    }
    return dmin(t12min, t1_2d);
}

/* localSolver.F90:195-289, node (iz, ix) 1-based. */
__device__ double init2(const Src2 &q, const Mesh2 &c, int sz, int sx, double tv,
                        double te, double tev, double t, double sref1, double sref2,
                        double sref3, int iz, int ix)
{
    const double sgnrz = (double)sz, sgnrx = (double)sx;
    double t1d = dmin(tv + c.dz * sref1, te + c.dx * sref2);
    double t1 = FK_HUGE, t2 = FK_HUGE, t3 = FK_HUGE;
    if (abs(iz - q.zsi) > q.eps || abs(ix - q.xsi) > q.eps) {
        if (tv <= te + c.dx * sref3 && te <= tv + c.dz * sref3 && te >= tev && tv >= tev) {
            double ta = tev + te - tv, tb = tev - te + tv;
            t1 = ((tb * c.dz2i + ta * c.dx2i) +
                  sqrt(4.0 * sref3 * sref3 * (c.dz2i + c.dx2i) -
                       c.dz2i * c.dx2i * (ta - tb) * (ta - tb))) /
                 (c.dz2i + c.dx2i);
        } else if ((te - tev) <= c.dz * c.dz * sref3 / sqrt(c.dx * c.dx + c.dz * c.dz) &&
                   te > tev) {
            double r = (te - tev) / c.dz;
            t2 = te + c.dx * sqrt(sref3 * sref3 - r * r);
        } else if ((tv - tev) <= c.dx * c.dx * sref3 / sqrt(c.dx * c.dx + c.dz * c.dz) &&
                   tv > tev) {
            double r = (tv - tev) / c.dx;
            t3 = tv + c.dz * sqrt(sref3 * sref3 - r * r);
        }
    } else {
        /* tAnaD (localSolver.F90:74-112) and the perturbations, used only by
         * the spherical operator near the source */
        double dz_ = ((double)iz - q.zsa) * c.dz, dx_ = ((double)ix - q.xsa) * c.dx;
        double d0 = dz_ * dz_ + dx_ * dx_;
        double t0c = 0.0, d0i_szero = 0.0;
        if (d0 > 0.0) {
            double sq = sqrt(d0);
            t0c = q.szero * sq;
            d0i_szero = q.szero / sq;
        }
        double tzc = d0i_szero * dz_, txc = d0i_szero * dx_;
        double tauv = tv - tana2(q, c, iz - sz, ix);
        double taue = te - tana2(q, c, iz, ix - sx);
        double tauev = tev - tana2(q, c, iz - sz, ix - sx);
        if (tv < te + c.dx * sref3 && te < tv + c.dz * sref3 && te >= tev && tv >= tev) {
            double ta = tauev + taue - tauv, tb = tauev - taue + tauv;
            double apoly = c.dz2i + c.dx2i;
            double bpoly = 4.0 * (sgnrx * txc * c.dxi + sgnrz * tzc * c.dzi) -
                           2.0 * (ta * c.dx2i + tb * c.dz2i);
            double cpoly = (ta * ta * c.dx2i) + (tb * tb * c.dz2i) -
                           4.0 * (sgnrx * txc * c.dxi * ta + sgnrz * tzc * c.dzi * tb) +
                           4.0 * (q.szero * q.szero - sref3 * sref3);
            double dpoly = bpoly * bpoly - 4.0 * apoly * cpoly;
            if (dpoly >= 0.0) t1 = 0.5 * (sqrt(dpoly) - bpoly) / apoly + t0c;
            if (t1 < tv || t1 < te) t1 = FK_HUGE;
        }
    }
    double t2d = dmin(dmin(t1, t2), t3);
    return dmin(dmin(t, t1d), t2d);
}

__device__ __forceinline__ void bar(int n)
{
    asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory");
}

struct Smem2 {
    Mesh2 mesh;
    double xres[2][kMaxWarps];
    double wmax[kMaxWarps];
};

template <bool INIT>
__device__ double sweep2(Smem2 &sm, double *ring, const Src2 &q, const fk_grid2d_t &g,
                         double *__restrict__ tt, const double *__restrict__ slow,
                         int sweep, int nthreads)
{
    const int nz = g.nz, nx = g.nx, zp = g.zp, zcp = g.zcp;
    const int sz = (sweep <= 2) ? 1 : -1;            /* localSolver.F90:160-193 */
    const int sx = (sweep == 1 || sweep == 3) ? 1 : -1;
    int loz = 1, lox = 1;
    if (INIT) {
        loz = (sz > 0) ? max(1, q.zsi - 1) : max(1, nz - q.zsi - 1);
        lox = (sx > 0) ? max(1, q.xsi - 1) : max(1, nx - q.xsi - 1);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = threadIdx.x;
    const int nblk = (nx + nthreads - 1) / nthreads;   /* column blocks */
    /* steps per block: the ring between blocks needs >= nthreads; one block needs no ring */
    const int zb = (nblk > 1 && nthreads > nz) ? nthreads : nz;
    const int nsteps = nblk * zb + nthreads - 1;
    /* The node and slowness loads of a thread's next item are issued one
     * step ahead: within a sweep only this thread writes its columns. */
    struct Item {
        double told, sUU, sUD, sDU;
        size_t idx;
        int iz, ix, b, il;
        bool valid, upd;
    };
    auto fetch = [&](int j, Item &f) {
        f.b = j >= 0 ? j / zb : -1;
        f.il = j - f.b * zb;
        const int xl = f.b * nthreads + t;
        f.valid = j >= 0 && f.b < nblk && xl < nx && f.il < nz;
        f.upd = f.valid && f.il >= loz && xl >= lox;
        if (!f.valid) return;
        f.ix = (sx > 0) ? xl : nx - 1 - xl;
        f.iz = (sz > 0) ? f.il : nz - 1 - f.il;
        f.idx = (size_t)f.ix * zp + f.iz;
        f.told = tt[f.idx];
        if (f.upd) {
            const int cxU = (sx > 0) ? f.ix - 1 : f.ix;
            const int cxD = min(max((sx > 0) ? f.ix : f.ix - 1, 0), nx - 2);
            const int czU = (sz > 0) ? f.iz - 1 : f.iz;
            const int czD = min(max((sz > 0) ? f.iz : f.iz - 1, 0), nz - 2);
            f.sUU = slow[(size_t)cxU * zcp + czU];
            f.sUD = slow[(size_t)cxD * zcp + czU]; /* z U, x D */
            f.sDU = slow[(size_t)cxU * zcp + czD]; /* z D, x U */
        }
    };
    Item nxt;
    fetch(-t, nxt);
    double r_last = FK_HUGE, te_last = FK_HUGE, dmax = 0.0;
    for (int s = 0; s < nsteps; ++s) {
        const Item cur = nxt;
        fetch(s + 1 - t, nxt);
        double te = __shfl_up_sync(0xffffffffu, r_last, 1);
        if (lane == 0 && warp > 0) te = sm.xres[(s + 1) & 1][warp - 1];
        if (t == 0) te = (cur.b > 0 && cur.il < nz) ? ring[cur.il] : FK_HUGE;
        double result = r_last;
        if (cur.valid) {
            const double told = cur.told;
            result = told;
            if (cur.upd) {
                const double s1 = dmin(cur.sUU, cur.sUD), s2 = dmin(cur.sUU, cur.sDU), s3 = cur.sUU;
                double tu;
                if (INIT)
                    tu = init2(q, sm.mesh, sz, sx, r_last, te, te_last, told, s1, s2, s3,
                               cur.iz + 1, cur.ix + 1);
                else
                    tu = noinit2(sm.mesh, r_last, te, te_last, s1, s2, s3);
                result = dmin(told, tu);
                if (result != told) {
                    tt[cur.idx] = result;
                    double d = fabs(result - told);
                    dmax = d > dmax ? d : dmax;
                }
            }
        }
        te_last = te;
        r_last = result;
        if (lane == 31) sm.xres[s & 1][warp] = result;
        if (t == nthreads - 1 && cur.b >= 0 && cur.b < nblk && cur.il < nz) ring[cur.il] = result;
        bar(nthreads);
    }
    return dmax;
}

__global__ void __launch_bounds__(kMaxThreads, 1)
solve2d_kernel(const fk_grid2d_t *__restrict__ grids, const fk_work2d_t *__restrict__ work,
               fk_result3d_t *__restrict__ results, double eps, int nsweep,
               double conv_tol, int max_pass)
{
    __shared__ Smem2 sm;
    extern __shared__ double ring2[];                 /* [nz]: last thread -> thread 0 of the next block */
    const fk_work2d_t w = work[blockIdx.x];
    const fk_grid2d_t g = grids[w.grid];
    const int nthreads = min(((g.nx + 31) / 32) * 32, (int)blockDim.x);
    if ((int)threadIdx.x >= nthreads) return;
    Src2 q;
    q.zsi = w.zsi; q.xsi = w.xsi; q.zsa = w.zsa; q.xsa = w.xsa; q.szero = w.szero;
    q.eps = eps; /* grid points, localSolver.F90:327 */
    if (threadIdx.x == 0) {
        Mesh2 &m = sm.mesh;
        m.dz = g.dz; m.dx = g.dx;
        m.dzi = 1.0 / g.dz; m.dxi = 1.0 / g.dx;
        m.dz2i = 1.0 / (g.dz * g.dz); m.dx2i = 1.0 / (g.dx * g.dx);
        m.dz2i_dx2i = m.dz2i * m.dx2i;
        m.dz2i_p_dx2i = m.dz2i + m.dx2i;
        m.dz2i_p_dx2i_inv = 1.0 / (m.dz2i + m.dx2i);
    }
    if (threadIdx.x < 2 * kMaxWarps) sm.xres[threadIdx.x / kMaxWarps][threadIdx.x % kMaxWarps] = FK_HUGE;
    double *tt = w.tt;
    const size_t nfield = (size_t)g.nx * g.zp;
    for (size_t e = threadIdx.x; e < nfield; e += nthreads) tt[e] = FK_HUGE;
    bar(nthreads);
    if (threadIdx.x < 4) { /* localSolver.F90:342-349 */
        const int di = threadIdx.x & 1, dj = threadIdx.x >> 1;
        tt[(size_t)(q.xsi - 1 + dj) * g.zp + (q.zsi - 1 + di)] =
            tana2(q, sm.mesh, q.zsi + di, q.xsi + dj);
    }
    __threadfence_block();
    bar(nthreads);
    for (int s = 1; s <= 4; ++s) sweep2<true>(sm, ring2, q, g, tt, g.slow, s, nthreads);
    const bool converge = conv_tol >= 0.0 && max_pass > 0;
    const int npasses = converge ? max_pass : nsweep;
    double res = 0.0;
    int ran = 0;
    for (int it = 0; it < npasses; ++it) {
        double d = 0.0;
        for (int s = 1; s <= 4; ++s) {
            double ds = sweep2<false>(sm, ring2, q, g, tt, g.slow, s, nthreads);
            d = ds > d ? ds : d;
        }
        for (int o = 16; o > 0; o >>= 1) {
            double v = __shfl_xor_sync(0xffffffffu, d, o);
            d = v > d ? v : d;
        }
        if ((threadIdx.x & 31) == 0) sm.wmax[threadIdx.x >> 5] = d;
        bar(nthreads);
        res = 0.0;
        for (int ww = 0; ww < (nthreads >> 5); ++ww) res = sm.wmax[ww] > res ? sm.wmax[ww] : res;
        bar(nthreads);
        ++ran;
        if (converge && res <= conv_tol) break;
    }
    if (threadIdx.x == 0) {
        results[blockIdx.x].residual = res;
        results[blockIdx.x].npass = ran;
        results[blockIdx.x].status = 0;
    }
}

/* ---- diagonal walk: grids up to 512 columns ------------------------------
 * A step of the walk above takes its nodes from a diagonal of the field: one
 * line per value in the [nx][zp] layout, index work and slowness minima in
 * every thread, and a root whose special cases branch, 1,050 cycles a step on
 * 201 x 201 (2.0 ms for 12 sweeps), where the chain of times itself (its
 * roots, comparisons and the hand-over to the next column) needs 290.  Here
 * everything but that chain is done beforehand, by kernels that use the whole
 * chip:
 *   items   what an update takes from the model, per sweep direction (shared
 *           by all sources), in rows of equal il + xl (logical z + logical x),
 *           so a step reads one contiguous row;
 *   field   two copies in rows: A of equal z + x (sweeps 1 and 4), B of equal
 *           z - x (sweeps 2 and 3).  A sweep walks its own copy; the sweeps
 *           before a change of copy (1 and 3, and the initialisation's) also
 *           store into the other one.
 * Rows hold 32-column multiples and padding rows follow, whose items leave a
 * time as it is, so the passes have no bounds to check.  A pass's step takes
 * 430 cycles (201 columns).  A whole call, 2 passes: one source on 201 x 201
 * 1.29 ms against 3.05 by the walk above, 256 sources on 151 x 301 3.0 ms
 * against 7.0. */
constexpr int kDiagCols = 512;     /* most columns: one thread each */
constexpr int kDiagAhead = 4;      /* steps from a load to its use */
constexpr int kDiagPad = 2 * kDiagAhead;   /* rows read past the last one */

struct Diag2 {
    int pitch, rows;               /* columns and rows of a plane, padding included */
    const int *odd;                /* the model may take roots out of sqrt64's range */
    const double2 *a12;            /* [4][rows][pitch]: dz s1, dx s2 */
    const double *s3;              /* [4][rows][pitch] */
    const double2 *lim;            /* [4][rows][pitch]: the edge operators' bounds (initialisation) */
    double *field;                 /* [nwork][2][rows][pitch] */
};

__host__ __device__ inline int diag_pitch(int nx) { return (nx + 31) / 32 * 32; }
__host__ __device__ inline int diag_rows(int nz, int nx) { return nz + nx - 1 + kDiagPad; }

/* Items of direction blockIdx.z: a node's (localSolver.F90:222-231); where
 * nothing is updated, additions that lose every comparison and a negative
 * slowness, whose bounds no time satisfies. */
__global__ void diag_items_kernel(fk_grid2d_t g, int pitch, int rows, double2 *a12, double2 *lim, double *s3,
                                  int *odd)
{
    const int xl = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y, dir = blockIdx.z;
    if (xl >= pitch) return;
    const int il = d - xl;
    const int sz = dir < 2 ? 1 : -1, sx = (dir & 1) ? -1 : 1;
    double2 a = make_double2(FK_HUGE, FK_HUGE), l = make_double2(-FK_HUGE, -FK_HUGE);
    double s = -1.0;
    if (il >= 1 && il < g.nz && xl >= 1 && xl < g.nx) {
        const int ix = (sx > 0) ? xl : g.nx - 1 - xl, iz = (sz > 0) ? il : g.nz - 1 - il;
        const int cxU = (sx > 0) ? ix - 1 : ix;
        const int cxD = min(max((sx > 0) ? ix : ix - 1, 0), g.nx - 2);
        const int czU = (sz > 0) ? iz - 1 : iz;
        const int czD = min(max((sz > 0) ? iz : iz - 1, 0), g.nz - 2);
        s = g.slow[(size_t)cxU * g.zcp + czU];
        a.x = g.dz * dmin(s, g.slow[(size_t)cxD * g.zcp + czU]);
        a.y = g.dx * dmin(s, g.slow[(size_t)cxU * g.zcp + czD]);
        const double diag = sqrt(g.dx * g.dx + g.dz * g.dz);
        l.x = g.dz * g.dz * s / diag;
        l.y = g.dx * g.dx * s / diag;
        /* the argument of a plane root whose conditions hold is at least
         * 4 s^2 / max(dz, dx)^2 */
        if (!(s > 1e-100 && s < 1e100 && g.dz > 1e-30 && g.dz < 1e30 && g.dx > 1e-30 && g.dx < 1e30)) *odd = 1;
    }
    const size_t i = ((size_t)dir * rows + d) * pitch + xl;
    a12[i] = a;
    lim[i] = l;
    s3[i] = s;
}

__global__ void diag_fill_kernel(double2 *f, size_t n)
{
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x)
        f[e] = make_double2(FK_HUGE, FK_HUGE);
}

/* Copy A back to the [nx][zp] field. */
__global__ void diag_out_kernel(fk_grid2d_t g, const fk_work2d_t *__restrict__ work, Diag2 dg)
{
    __shared__ double tile[32][33];
    const double *A = dg.field + (size_t)blockIdx.z * 2 * dg.rows * dg.pitch;
    double *tt = work[blockIdx.z].tt;
    const int x0 = blockIdx.x * 32, z0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int x = x0 + threadIdx.x, z = z0 + i;
        if (x < g.nx && z < g.nz) tile[i][threadIdx.x] = A[(size_t)(z + x) * dg.pitch + x];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int x = x0 + i, z = z0 + threadIdx.x;
        if (x < g.nx && z < g.nz) tt[(size_t)x * g.zp + z] = tile[threadIdx.x][i];
    }
}

/* tAnaD and tAna (localSolver.F90:36-112) of a node near the source. */
struct Near2 {
    double ana;          /* tAna */
    double t0c, tzc, txc;
};

__device__ __forceinline__ Near2 near_node(const Src2 &q, const Mesh2 &c, int iz, int ix)
{
    double dz_ = ((double)iz - q.zsa) * c.dz, dx_ = ((double)ix - q.xsa) * c.dx;
    double d0 = dz_ * dz_ + dx_ * dx_;
    double t0c = 0.0, d0i_szero = 0.0;
    if (d0 > 0.0) {
        double sq = sqrt(d0);
        t0c = q.szero * sq;
        d0i_szero = q.szero / sq;
    }
    return {tana2(q, c, iz, ix), t0c, d0i_szero * dz_, d0i_szero * dx_};
}

/* The nodes within kNear of the source and their upwind ones, evaluated once
 * per solve where eps allows (the roots, hypotenuses and quotients would
 * otherwise stand in the chain of every initialisation sweep). */
constexpr int kNear = 6, kNearN = 2 * kNear + 3;

struct SmemDiag {
    Mesh2 mesh;
    Src2 src;
    int near_cells;                      /* floor(eps) */
    bool have_near;
    double wmax[kMaxWarps];
    double res[2][kDiagCols + 1];        /* a step's results, by parity; slot 0: left of column 0 */
    Near2 near[kNearN][kNearN];
};

/* localSolver.F90:74-112, :232-289: the spherical operator near the source
 * (few nodes: kept out of the walk's registers), node (iz, ix) 1-based. */
__device__ __noinline__ double near2(const SmemDiag &sm, int sz, int sx, double tv, double te, double tev,
                                     double sref3, int iz, int ix)
{
    const Src2 &q = sm.src;
    const Mesh2 &c = sm.mesh;
    const double sgnrz = (double)sz, sgnrx = (double)sx;
    double t1 = FK_HUGE;
    if (tv < te + c.dx * sref3 && te < tv + c.dz * sref3 && te >= tev && tv >= tev) {
        Near2 n;
        double av, ae, aev;
        if (sm.have_near) {
            const int i = iz - q.zsi + kNear + 1, j = ix - q.xsi + kNear + 1;
            n = sm.near[i][j];
            av = sm.near[i - sz][j].ana;
            ae = sm.near[i][j - sx].ana;
            aev = sm.near[i - sz][j - sx].ana;
        } else {
            n = near_node(q, c, iz, ix);
            av = tana2(q, c, iz - sz, ix);
            ae = tana2(q, c, iz, ix - sx);
            aev = tana2(q, c, iz - sz, ix - sx);
        }
        double tauv = tv - av, taue = te - ae, tauev = tev - aev;
        double ta = tauev + taue - tauv, tb = tauev - taue + tauv;
        double apoly = c.dz2i + c.dx2i;
        double bpoly = 4.0 * (sgnrx * n.txc * c.dxi + sgnrz * n.tzc * c.dzi) -
                       2.0 * (ta * c.dx2i + tb * c.dz2i);
        double cpoly = (ta * ta * c.dx2i) + (tb * tb * c.dz2i) -
                       4.0 * (sgnrx * n.txc * c.dxi * ta + sgnrz * n.tzc * c.dzi * tb) +
                       4.0 * (q.szero * q.szero - sref3 * sref3);
        double dpoly = bpoly * bpoly - 4.0 * apoly * cpoly;
        if (dpoly >= 0.0) t1 = 0.5 * (sqrt(dpoly) - bpoly) / apoly + n.t0c;
        if (t1 < tv || t1 < te) t1 = FK_HUGE;
    }
    return t1;
}

/* The root on the chain: ODD for models whose roots may leave sqrt64's range. */
template <bool ODD>
__device__ __forceinline__ double root2(double x) { return ODD ? sqrt(x) : fk64::sqrt64(x); }

/* localSolver.F90:195-289 away from the source: one of three operators
 * applies (the plane one, or one of the edges' when it does not).  Their
 * roots' arguments are selected first, so the chain holds one square root;
 * an edge operator's may be zero. */
template <bool ODD>
__device__ __forceinline__ double far2(const Mesh2 &c, double tv, double te, double tev, double a1, double a2, double s3,
                                       double limz, double limx)
{
    const double bz = c.dz * s3, bx = c.dx * s3;
    const double t1d = dmin(tv + a1, te + a2);
    const double dte = te - tev, dtv = tv - tev;
    const bool plane = tv <= te + bx && te <= tv + bz && te >= tev && tv >= tev;
    const bool ez = !plane && dte <= limz && te > tev;
    const bool ex = !plane && !ez && dtv <= limx && tv > tev;
    const double ta = tev + te - tv, tb = tev - te + tv, tab = ta - tb;
    const double r = fk64::div64(ez ? dte : dtv, ez ? c.dz : c.dx, ez ? c.dzi : c.dxi);
    const double arg = plane ? 4.0 * s3 * s3 * c.dz2i_p_dx2i - c.dz2i_dx2i * tab * tab : s3 * s3 - r * r;
    double root = root2<ODD>(arg);
    if (!ODD && (ez || ex) && !fk64::sqrt64_ok(arg)) root = sqrt(arg);
    const double t1 = fk64::div64((tb * c.dz2i + ta * c.dx2i) + root, c.dz2i_p_dx2i, c.dz2i_p_dx2i_inv);
    const double t2 = (ez ? te : tv) + (ez ? c.dx : c.dz) * root;
    const double t2d = plane ? t1 : (ez || ex) ? t2 : FK_HUGE;
    return dmin(t1d, t2d);
}

/* One sweep: thread t walks the t-th column of the sweep's box and the column
 * and row before it (the whole grid in the passes), one position behind
 * thread t - 1.  own, other: the field copies.  Returns max |dt|. */
template <bool INIT, bool ODD>
__device__ __forceinline__ double diag_sweep(SmemDiag &sm, const Mesh2 &c, const fk_grid2d_t &g, const Diag2 &dg,
                                             double *A, double *B, int sweep)
{
    const int nz = g.nz, nx = g.nx, pitch = dg.pitch, t = threadIdx.x;
    const int sz = (sweep <= 2) ? 1 : -1;            /* localSolver.F90:160-193 */
    const int sx = (sweep == 1 || sweep == 3) ? 1 : -1;
    int loz = 1, lox = 1;
    if (INIT) {
        const int zsi = sm.src.zsi, xsi = sm.src.xsi;   /* solver2D.F90:825-867 */
        loz = (sz > 0) ? max(1, zsi - 1) : max(1, nz - zsi - 1);
        lox = (sx > 0) ? max(1, xsi - 1) : max(1, nx - xsi - 1);
    }
    const int xl = lox - 1 + t;
    const bool col = xl < nx;
    const int x = (sx > 0) ? xl : max(nx - 1 - xl, 0);
    const int d0 = loz - 1 + lox - 1;                /* the first step's logical row */
    const int nsteps = nz + nx - 1 - d0;
    /* copy A's rows z + x ascend with the logical row in sweep 1 and descend in
     * sweep 4, copy B's rows z - x + nx - 1 in sweeps 2 and 3 */
    const bool famA = sweep == 1 || sweep == 4;
    double *const own = famA ? A : B, *const other = famA ? B : A;
    const int row0 = (sz > 0) ? d0 : nz + nx - 2 - d0;
    const double *pf = own + (size_t)row0 * pitch + x;          /* times, AH steps ahead */
    double *ps = own + (size_t)row0 * pitch + x;                /* times, this step */
    const ptrdiff_t dp = (sz > 0) ? pitch : -pitch;
    /* the other copy's row of this column's position il = loz - 1 - t (step 0) */
    const bool both = INIT ? sweep < 4 : (sweep == 1 || sweep == 3);
    const int il0 = loz - 1 - t;
    const int iz0 = (sz > 0) ? il0 : nz - 1 - il0;
    double *po = other + (ptrdiff_t)(famA ? iz0 + nx - 1 - x : iz0 + x) * pitch + x;
    const size_t plane = (size_t)(2 * (sz < 0) + (sx < 0)) * dg.rows * pitch + (size_t)d0 * pitch + min(xl, pitch - 1);
    const double2 *pa = dg.a12 + plane;
    const double *p3 = dg.s3 + plane;
    const double2 *pl = dg.lim + plane;
    const int near = sm.near_cells;                  /* |iz - zsi|, |ix - xsi| of the spherical operator */
    const int zsi = sm.src.zsi, xsi = sm.src.xsi;
    struct Slot {
        double2 a, lim;
        double s3, told;
    };
    constexpr int AH = INIT ? 2 : kDiagAhead;        /* the initialisation's operators need the registers */
    Slot slot[AH];
    int left = nsteps;                               /* rows of times still to load */
    auto load = [&](Slot &f) {
        f.a = __ldg(pa);
        f.s3 = __ldg(p3);
        if (INIT) {
            f.lim = __ldg(pl);
            pl += pitch;
        }
        f.told = FK_HUGE;
        if (left > 0 && (!INIT || col)) f.told = *pf;
        --left;
        pa += pitch;
        p3 += pitch;
        pf += dp;
    };
#pragma unroll
    for (int u = 0; u < AH; ++u) load(slot[u]);
    sm.res[0][t + 1] = sm.res[1][t + 1] = FK_HUGE;
    if (t == 0) sm.res[0][0] = sm.res[1][0] = FK_HUGE;
    __syncthreads();
    const double P4 = 4.0 * c.dz2i_p_dx2i;           /* (4 s s) P = (s s) (4 P): a power of two */
    double r_last = FK_HUGE, te_last = FK_HUGE, dmax = 0.0;
    for (int s0 = 0; s0 < nsteps; s0 += AH) {
#pragma unroll
        for (int u = 0; u < AH; ++u) {
            const Slot w = slot[u];
            load(slot[u]);
            const int k = s0 + u - t;                /* position in the walk */
            const double tv = r_last, tev = te_last, te = sm.res[(u + 1) & 1][t];
            double result;
            if (INIT) {
                const bool upd = k >= 1 && t >= 1 && k < nz - loz + 1 && col;
                double tu = far2<ODD>(c, tv, te, tev, w.a.x, w.a.y, w.s3, w.lim.x, w.lim.y);
                const int il = loz - 1 + k;
                const int iz = (sz > 0) ? il + 1 : nz - il, ix = x + 1;   /* 1-based */
                if (upd && abs(iz - zsi) <= near && abs(ix - xsi) <= near)
                    tu = dmin(dmin(tv + w.a.x, te + w.a.y), near2(sm, sz, sx, tv, te, tev, w.s3, iz, ix));
                result = upd ? dmin(w.told, tu) : w.told;
                if (upd && result != w.told) {
                    *ps = result;
                    if (both) *po = result;
                }
            } else {
                /* localSolver.F90:123-158, straight-line: a candidate that its
                 * conditions reject may be NaN, the select drops it */
                const double bz = c.dz * w.s3, bx = c.dx * w.s3, q = (w.s3 * w.s3) * P4;
                const double temtv = te - tv;
                const double t12min = dmin(tv + w.a.x, te + w.a.y);
                const double ta = tev + temtv, tb = tev - temtv, tab = ta - tb;
                const double t1_2d = ((tb * c.dz2i + ta * c.dx2i) + root2<ODD>(q - c.dz2i_dx2i * (tab * tab))) *
                                     c.dz2i_p_dx2i_inv;
                const double tu = (temtv < bz && -temtv < bx) ? dmin(t12min, t1_2d) : t12min;
                result = dmin(w.told, tu);
                if (result != w.told) {
                    *ps = result;
                    const double d = w.told - result;
                    dmax = d > dmax ? d : dmax;
                }
                if (both && (unsigned)k < (unsigned)nz && col) *po = result;
            }
            sm.res[u & 1][t + 1] = result;
            te_last = te;
            r_last = result;
            ps += dp;
            po += dp;
            __syncthreads();
        }
    }
    return dmax;
}

template <bool ODD>
__device__ __forceinline__ void diag_solve(SmemDiag &sm, const fk_grid2d_t &g, const Diag2 &dg, double *A, double *B,
                                           fk_result3d_t *result, int nsweep)
{
    const Mesh2 mesh = sm.mesh;
#pragma unroll 1
    for (int s = 1; s <= 4; ++s) diag_sweep<true, ODD>(sm, mesh, g, dg, A, B, s);
    double d = 0.0;
#pragma unroll 1
    for (int it = 0; it < nsweep; ++it) {
        d = 0.0;
#pragma unroll 1
        for (int s = 1; s <= 4; ++s) {
            const double ds = diag_sweep<false, ODD>(sm, mesh, g, dg, A, B, s);
            d = ds > d ? ds : d;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double v = __shfl_xor_sync(0xffffffffu, d, o);
        d = v > d ? v : d;
    }
    if ((threadIdx.x & 31) == 0) sm.wmax[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        double res = 0.0;
        for (int w = 0; w < (int)blockDim.x >> 5; ++w) res = sm.wmax[w] > res ? sm.wmax[w] : res;
        result->residual = res;
        result->npass = nsweep;
        result->status = 0;
    }
}

/* MAXT threads at most, PER CTAs to an SM: more sources than SMs share them
 * (the chain leaves issue slots), where the registers allow it. */
template <int MAXT, int PER>
__global__ void __launch_bounds__(MAXT, PER)
diag_solve_kernel(fk_grid2d_t g, const fk_work2d_t *__restrict__ work, fk_result3d_t *__restrict__ results, Diag2 dg,
                  double eps, int nsweep)
{
    __shared__ SmemDiag sm;
    const fk_work2d_t w = work[blockIdx.x];
    double *const A = dg.field + (size_t)blockIdx.x * 2 * dg.rows * dg.pitch, *const B = A + (size_t)dg.rows * dg.pitch;
    const int nthreads = blockDim.x, t = threadIdx.x;
    Src2 q;
    q.zsi = w.zsi; q.xsi = w.xsi; q.zsa = w.zsa; q.xsa = w.xsa; q.szero = w.szero;
    q.eps = eps; /* grid points, localSolver.F90:327 */
    if (t == 0) {
        Mesh2 &m = sm.mesh;
        m.dz = g.dz; m.dx = g.dx;
        m.dzi = 1.0 / g.dz; m.dxi = 1.0 / g.dx;
        m.dz2i = 1.0 / (g.dz * g.dz); m.dx2i = 1.0 / (g.dx * g.dx);
        m.dz2i_dx2i = m.dz2i * m.dx2i;
        m.dz2i_p_dx2i = m.dz2i + m.dx2i;
        m.dz2i_p_dx2i_inv = 1.0 / (m.dz2i + m.dx2i);
        sm.src = q;
        sm.near_cells = eps < 0.0 ? -1 : eps < 1e9 ? (int)eps : 1000000000;
        sm.have_near = eps <= (double)kNear;
    }
    __syncthreads();
    const bool odd = *dg.odd != 0;
    for (int e = t; e < kNearN * kNearN; e += nthreads)
        sm.near[e / kNearN][e % kNearN] =
            near_node(q, sm.mesh, q.zsi + e / kNearN - kNear - 1, q.xsi + e % kNearN - kNear - 1);
    if (t < 4) { /* localSolver.F90:342-349 */
        const int di = t & 1, dj = t >> 1, z = q.zsi - 1 + di, x = q.xsi - 1 + dj;
        const double v = tana2(q, sm.mesh, q.zsi + di, q.xsi + dj);
        A[(size_t)(z + x) * dg.pitch + x] = v;
        B[(size_t)(z + g.nx - 1 - x) * dg.pitch + x] = v;
    }
    __threadfence_block();
    __syncthreads();
    if (odd) diag_solve<true>(sm, g, dg, A, B, results + blockIdx.x, nsweep);
    else diag_solve<false>(sm, g, dg, A, B, results + blockIdx.x, nsweep);
}

} // namespace

/* Bytes of the diagonal walk's model planes and of one source's field
 * copies; false where it does not apply: more columns than threads, or model
 * planes above 1 GiB (the walk above reads the model in place). */
extern "C" int fk2d_diag_bytes(int nz, int nx, size_t *model, size_t *source)
{
    const size_t plane = (size_t)diag_rows(nz, nx) * diag_pitch(nx);
    *model = 256 + plane * 4 * (2 * sizeof(double2) + sizeof(double));
    *source = plane * 2 * sizeof(double);
    return nx <= kDiagCols && diag_rows(nz, nx) <= 65535 && *model <= ((size_t)1 << 30);
}

/* nsweep passes over every work item of one grid; scratch holds the model
 * planes, then nwork sources' field copies.  set_model: build the planes (they
 * stay in scratch for further calls on the same grid and model). */
extern "C" int fk2d_solve_diag(const fk_grid2d_t *grid, const fk_work2d_t *work, fk_result3d_t *results, int nwork,
                               double eps, int nsweep, void *scratch, int set_model, cudaStream_t stream)
{
    if (nwork <= 0) return 0;
    const fk_grid2d_t g = *grid;
    Diag2 dg;
    dg.pitch = diag_pitch(g.nx);
    dg.rows = diag_rows(g.nz, g.nx);
    const size_t plane = (size_t)dg.rows * dg.pitch;
    int *odd = (int *)scratch;
    double2 *a12 = (double2 *)((char *)scratch + 256);
    double2 *lim = a12 + 4 * plane;
    double *s3 = (double *)(lim + 4 * plane);
    dg.odd = odd;
    dg.a12 = a12;
    dg.lim = lim;
    dg.s3 = s3;
    dg.field = s3 + 4 * plane;
    if (set_model) {
        cudaError_t e = cudaMemsetAsync(odd, 0, sizeof(int), stream);
        if (e != cudaSuccess) return (int)e;
        diag_items_kernel<<<dim3((dg.pitch + 127) / 128, dg.rows, 4), 128, 0, stream>>>(g, dg.pitch, dg.rows, a12, lim,
                                                                                      s3, odd);
    }
    const size_t n2 = (size_t)nwork * plane;          /* double2 of both copies */
    diag_fill_kernel<<<(unsigned)(n2 / 512 + 1 < 148 * 16 ? n2 / 512 + 1 : 148 * 16), 256, 0, stream>>>(
        (double2 *)dg.field, n2);
    /* 256 sources on 151 x 301: 3.0 ms with two CTAs to an SM (102 registers),
     * 4.2 with one (128); 200 on 200 x 360 4.3 and 5.2 (80 registers), 256 on
     * 250 x 400 6.2 and 6.9 (72), but 256 on 400 x 500 11.5 and 10.7 (64); one
     * source on 201 x 201 is 2 % faster with 176 registers than with 128 */
    const bool share = nwork > 148;
    auto *kernel = dg.pitch <= 256   ? (share ? diag_solve_kernel<256, 2> : diag_solve_kernel<256, 1>)
                   : !share          ? diag_solve_kernel<kDiagCols, 1>
                   : dg.pitch <= 320 ? diag_solve_kernel<320, 2>
                   : dg.pitch <= 384 ? diag_solve_kernel<384, 2>
                   : dg.pitch <= 448 ? diag_solve_kernel<448, 2>
                                     : diag_solve_kernel<kDiagCols, 1>;
    kernel<<<nwork, dg.pitch, 0, stream>>>(g, work, results, dg, eps, nsweep);
    for (int w0 = 0; w0 < nwork; w0 += 65535) {
        Diag2 d1 = dg;
        d1.field = dg.field + (size_t)w0 * 2 * plane;
        const int n = nwork - w0 < 65535 ? nwork - w0 : 65535;
        diag_out_kernel<<<dim3((g.nx + 31) / 32, (g.nz + 31) / 32, n), dim3(32, 8), 0, stream>>>(g, work + w0, d1);
    }
    return (int)cudaGetLastError();
}

extern "C" int fk2d_solve(int fsm, const fk_grid2d_t *grids, const fk_work2d_t *work,
                          fk_result3d_t *results, int nwork, int max_nx, int max_nz, double eps,
                          int nsweep, double conv_tol, int max_pass, cudaStream_t stream)
{
    (void)fsm; /* same dependency graph, same result: see the file comment */
    if (nwork <= 0) return 0;
    const int nthreads = min(((max_nx + 31) / 32) * 32, kMaxThreads);
    const size_t smem = sizeof(double) * (size_t)(max_nz > 1 ? max_nz : 1);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(solve2d_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    solve2d_kernel<<<nwork, nthreads, smem, stream>>>(grids, work, results, eps, nsweep,
                                                      conv_tol, max_pass);
    return (int)cudaGetLastError();
}
