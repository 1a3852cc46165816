/*
 * tile3d.cu -- 3D solve of few sources on grids whose tiles fit the chip at
 * once (the whole field in shared memory).
 *
 * With few sources the slab schedule (row3d_impl.cuh) is bound by its chain:
 * a slab walks its column blocks one after the other, 128 columns x 128
 * positions in 512 steps, and each of the 32 slabs of a sweep starts some
 * 20 steps behind the one before; a converged 128^3 solve spends 430 us a
 * sweep with 32 blocks busy.  Here a block owns a tile of 16 x 8 (x, y)
 * columns over all z for the whole solve, every column has a thread, and a
 * sweep is one wavefront over all tiles: nx + ny + nz steps and a hand-over
 * per tile.  Field and slowness of the tile stay in shared memory from the
 * first sweep to the last (loaded and stored once), so a step has no global
 * access but the tile's edges.
 *
 * Step t of a block: the thread of logical column (lx, ly) updates position
 * t - lx - ly.  Results go to a plane in shared memory (4 steps deep, a border
 * row and column for the upwind tiles' edges); te and tn are the neighbours'
 * results of step t - 1, ten the diagonal neighbour's of step t - 2, and tv,
 * tev, tnv, tnve the thread's own te, tn, ten and result of the step before.
 *
 * Edges travel through global memory as words {sweep + 1, value bits}: the tag
 * makes the value its own flag, so there is no fence and no counter.  A fifth
 * warp polls the words of the upwind tiles, four steps ahead, and writes them
 * into the plane's border.  Rows of words follow the producer's steps, so a
 * step's words are contiguous on both sides.  In the passes two buffers by the
 * sweep's parity suffice: x changes direction in every sweep and y in every
 * other one, so before a tile writes a buffer again it has waited, directly or
 * through the tile beside it, for each reader (the diagonal one included) to
 * be in a later sweep.  In the initialisation a tile before the source's box
 * waits for nobody, so its sweeps and the first two of the passes have buffers
 * of their own.  The tag's upper bits count launches, so buffers need no
 * clearing.
 *
 * Measured (one source): 128^3 in FP32, a pass's sweep 108 to 114 us against 430
 * and more, converged after 3, 7 and 9 passes 4.1, 7.7 and 9.6 ms a call against
 * 20.8, 41 and 50 (slabs, knobs 0, 1, 0, 0); 41 x 53 x 47 in FP64 2.3 ms a call
 * against 7.6.  A step takes 400 cycles in FP32 (bound by its 145
 * instructions at one warp to a scheduler) and 1,100 in FP64 (160 FP64
 * instructions, which one warp issues every 4.4 cycles); a hand-over to the
 * next tile costs 6 to 7 steps.
 *
 * All blocks wait for one another, so the launch is cooperative; every wait
 * has a poll limit, after which the error word is set and all blocks return.
 * Updates, their order and their arithmetic are those of the slab schedule:
 * the fields are the same bits.  Compiled without multiply-add contraction
 * (the FP64 stencils round as the CPU algorithm does).
 */
#include "slab3d_common.cuh"
#include "fp64.cuh"

namespace fk3tl {
using fk3::Mesh;
using fk3::Src;
using fk3::rmin;
using fk3::rmax;

constexpr int TX = 16, TY = 8, NC = TX * TY;   /* columns of a tile: 2 x 2 warps of 8 x 4 */
constexpr int NT = NC + 32;                    /* and the edge warp */
constexpr int PW = 24;                         /* plane row: 8 x 4 lanes hit 32 banks */
constexpr int EW = TX + TY;                    /* edge words of a step: TY of the x edge, TX of the y edge */
constexpr int GUARD = 32;                      /* values before and after the tile that idle lanes may read */
constexpr int EBUF = 10;                       /* edge buffers: sweeps 0-9, then by parity */
constexpr int AHEAD = 4;                       /* steps from an edge word's load to its use */

struct Params {
    const fk_grid3d_t *grids;
    const fk_work3d_t *work;
    const int2 *tiles;          /* this launch's tiles: {work, bx | by << 16} */
    const int *tile0;           /* per work item: its first tile among all works' */
    int tile_base;              /* number of the launch's first tile among all works' */
    unsigned long long *edge;   /* [tile][EBUF][rows][EW] words (FP64: two planes of words) */
    const unsigned *epoch;      /* counts launches */
    int rows;
    int *error;
    unsigned long long *resid;  /* [nwork][npass] */
    int *pass_tiles;            /* [nwork][npass]: tiles done with the pass */
    int *conv_pass;             /* [nwork] */
    int npass;
    double eps, conv_tol;
    long long spin_limit;
};

/* Column pitch in shared memory: 5 mod 8, which spreads the 8 x 4 skewed
 * columns of a warp over 32 banks in half of the sweeps, 16 in the others. */
__host__ __device__ inline int pitch5(int n) { return n + ((5 - n) & 7); }

template <typename R>
__host__ __device__ inline size_t tile_bytes(int nz)
{
    return sizeof(R) * ((size_t)NC * pitch5(nz) + (size_t)(TX + 1) * (TY + 1) * pitch5(nz + 1) + 2 * GUARD);
}

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

/* Stores under a predicate (no branch in the walk). */
__device__ __forceinline__ void st_word_if(bool p, unsigned long long *a, unsigned long long v)
{
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q st.relaxed.gpu.global.u64 [%0], %1; }" ::"l"(a), "l"(v),
                 "r"((int)p)
                 : "memory");
}
__device__ __forceinline__ void st_shared_if(bool p, unsigned a, float v)
{
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q st.shared.f32 [%0], %1; }" ::"r"(a), "f"(v), "r"((int)p)
                 : "memory");
}
__device__ __forceinline__ void st_shared_if(bool p, unsigned a, double v)
{
    asm volatile("{ .reg .pred q; setp.ne.s32 q, %2, 0; @q st.shared.f64 [%0], %1; }" ::"r"(a), "d"(v), "r"((int)p)
                 : "memory");
}
__device__ __forceinline__ float ld_shared(unsigned a, float)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double ld_shared(unsigned a, double)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}

/* An edge value: one tagged word per 32 bits of it, `plane` words apart. */
template <typename R> struct Word;
template <> struct Word<float> {
    unsigned long long a;
    __device__ void load(const unsigned long long *p, size_t) { a = ld_word(p); }
    __device__ bool ok(unsigned tag) const { return (unsigned)(a >> 32) == tag; }
    __device__ float value() const { return __uint_as_float((unsigned)a); }
    static __device__ __forceinline__ void store(bool on, unsigned long long *p, size_t, unsigned tag, float v)
    {
        st_word_if(on, p, (unsigned long long)tag << 32 | __float_as_uint(v));
    }
};
template <> struct Word<double> {
    unsigned long long a, b;
    __device__ void load(const unsigned long long *p, size_t plane)
    {
        a = ld_word(p);
        b = ld_word(p + plane);
    }
    __device__ bool ok(unsigned tag) const { return (unsigned)(a >> 32) == tag && (unsigned)(b >> 32) == tag; }
    __device__ double value() const { return __hiloint2double((int)(unsigned)b, (int)(unsigned)a); }
    static __device__ __forceinline__ void store(bool on, unsigned long long *p, size_t plane, unsigned tag, double v)
    {
        st_word_if(on, p, (unsigned long long)tag << 32 | (unsigned)__double2loint(v));
        st_word_if(on, p + plane, (unsigned long long)tag << 32 | (unsigned)__double2hiint(v));
    }
};

template <typename R>
struct Smem {
    R plane[4][TY + 1][PW];      /* [step mod 4][ly + 1][lx + 1] */
    Src src;
    Mesh<double> mesh64;
    double max[4];
    unsigned epoch;
    int dead, stop;
};

/* Spherical stencil near the source (localSolver.F90:538-751, tmin <= eps):
 * few nodes, kept out of the walk's registers. */
__device__ __noinline__ double near3(const Src &q, const Mesh<double> &m, double tv, double te, double tn, double tev,
                                     double ten, double tnv, double tnve, double told, double s1, double s2, double s3,
                                     double s4, double s5, double s6, double s7, int i, int j, int k, int sz, int sx,
                                     int sy)
{
    return fk3::init_node<double>(q, m, false, tv, te, tn, tev, ten, tnv, tnve, told, s1, s2, s3, s4, s5, s6, s7, i, j,
                                  k, sz, sx, sy);
}

/* FP64 plane-wave stencils in the reference's operand order, straight-line:
 * INIT in that of fteik_localSolver_init64fF's Cartesian branches
 * (localSolver.F90:625-732), else noInit64fF's (:384-534).  The four roots are
 * branch-free; arguments that an accepted candidate may not give sqrt64 are
 * reported. */
template <bool INIT>
__device__ __forceinline__ double cart64(const Mesh<double> &c, double tv, double te, double tn, double tev, double ten,
                                         double tnv, double tnve, double s1, double s2, double s3, double s4, double s5,
                                         double s6, double s7, double told, bool &odd)
{
    const double HUGEV = FK_HUGE;
    double m = rmin(rmin(tv + c.dz * s1, te + c.dx * s2), tn + c.dy * s3);
    const double temtv = te - tv, tvmtn = tv - tn, temtn = te - tn;
    const double zxa = INIT ? tev + te - tv : tev + temtv, zxb = INIT ? tev - te + tv : tev - temtv;
    const double zya = INIT ? tv - tn + tnv : tvmtn + tnv, zyb = INIT ? tn - tv + tnv : -tvmtn + tnv;
    const double xya = INIT ? te - tn + ten : temtn + ten, xyb = INIT ? tn - te + ten : -temtn + ten;
    const double zx = zxa - zxb, zy = zya - zyb, xy = xya - xyb;
    const double q_zx = 4.0 * (s4 * s4) * c.dz2i_p_dx2i - c.dz2i_dx2i * (zx * zx);
    const double q_zy = 4.0 * (s5 * s5) * c.dz2i_p_dy2i - c.dz2i_dy2i * (zy * zy);
    const double q_xy = 4.0 * (s6 * s6) * c.dx2i_p_dy2i - c.dx2i_dy2i * (xy * xy);
    const double ta = te + 0.5 * (-tn + ten - tv + tev) - tnv + tnve;
    const double tb = tv + 0.5 * (-tn + tnv - te + tev) - ten + tnve;
    const double tc = tn + 0.5 * (-te + ten - tv + tnv) - tev + tnve;
    const double tab = ta - tb, tbc = tb - tc, tac = ta - tc;
    const double t2 = (s7 * s7) * c.dsum_nine;
    const double t3 = c.dz2dx2 * (tab * tab) + c.dz2dy2 * (tbc * tbc) + c.dx2dy2 * (tac * tac);
    const double q_3 = t2 - t3;
    const double t_zx = ((zxb * c.dz2i + zxa * c.dx2i) + fk64::sqrt64(q_zx)) * c.dz2i_p_dx2i_inv;
    const double t_zy = ((zya * c.dz2i + zyb * c.dy2i) + fk64::sqrt64(q_zy)) * c.dz2i_p_dy2i_inv;
    const double t_xy = ((xya * c.dx2i + xyb * c.dy2i) + fk64::sqrt64(q_xy)) * c.dx2i_p_dy2i_inv;
    const double r_3 = q_3 > 0.0 ? fk64::sqrt64(q_3) : 0.0;
    const double t_3 = (tb * c.dz2i + ta * c.dx2i + tc * c.dy2i + r_3) * c.dsumi;
    bool zxok, zyok, xyok;
    if (INIT) {
        zxok = tv < te + c.dx * s4 && te < tv + c.dz * s4;
        zyok = tv < tn + c.dy * s5 && tn < tv + c.dz * s5;
        xyok = te < tn + c.dy * s6 && tn < te + c.dx * s6;
    } else {
        zxok = temtv < c.dz * s4 && -temtv < c.dx * s4;
        zyok = tvmtn < c.dy * s5 && -tvmtn < c.dz * s5;
        xyok = temtn < c.dy * s6 && -temtn < c.dx * s6;
    }
    m = zxok ? rmin(m, t_zx) : m;
    m = zyok ? rmin(m, t_zy) : m;
    m = xyok ? rmin(m, t_xy) : m;
    const double tmax = rmax(rmax(tv, te), tn);
    const bool ok3 = m > tmax && t2 >= t3;
    odd = (zxok && !fk64::sqrt64_ok(q_zx)) || (zyok && !fk64::sqrt64_ok(q_zy)) || (xyok && !fk64::sqrt64_ok(q_xy)) ||
          (ok3 && q_3 != 0.0 && !fk64::sqrt64_ok(q_3));
    return rmin(told, rmin(ok3 ? t_3 : HUGEV, m));
}

__device__ __noinline__ double cart64_any(bool init, const Mesh<double> &m, double tv, double te, double tn, double tev,
                                          double ten, double tnv, double tnve, double s1, double s2, double s3,
                                          double s4, double s5, double s6, double s7, double told)
{
    if (init) {
        Src q = {};
        return fk3::init_node<double>(q, m, true, tv, te, tn, tev, ten, tnv, tnve, told, s1, s2, s3, s4, s5, s6, s7, 1, 1,
                                      1, 1, 1, 1);
    }
    return fk3::noinit<double>(m, tv, te, tn, tev, ten, tnv, tnve, s1, s2, s3, s4, s5, s6, s7, told);
}

/* What a block knows of its tile. */
struct Tile {
    int bx, by, ntx, nty, x0, y0, w, h;
    int tile;                    /* among the launch's */
    int work0;                   /* first tile of its work item among the launch's */
};

/* One sweep of a tile (see the file comment). */
template <typename R, bool INIT, bool CONV>
__device__ __forceinline__ void tile_sweep(const Params &P, Smem<R> &sm, R *F, const R *S, const fk_grid3d_t &g,
                                           const Tile &tl, const Mesh<R> &mesh, int s, double &dmax)
{
    const int nz = g.nz, nx = g.nx, ny = g.ny;
    const int zpf = pitch5(nz), zps = pitch5(nz + 1);
    const int s0 = s % 8;
    const int sz = (s0 < 4) ? 1 : -1;
    const int sx = (s0 % 2 == 0) ? 1 : -1;
    const int sy = ((s0 / 2) % 2 == 0) ? 1 : -1;
    int loz = 1, lox = 1, loy = 1;
    if (INIT) { /* solver3D.F90:493-565, flipped bound clamped to the grid */
        loz = (sz > 0) ? max(1, sm.src.zsi - 1) : max(1, nz - sm.src.zsi - 1);
        lox = (sx > 0) ? max(1, sm.src.xsi - 1) : max(1, nx - sm.src.xsi - 1);
        loy = (sy > 0) ? max(1, sm.src.ysi - 1) : max(1, ny - sm.src.ysi - 1);
    }
    const int Z = nz - loz + 1;                      /* positions: logical z loz - 1 .. nz - 1 */
    const int xl0 = (sx > 0) ? tl.x0 : nx - tl.x0 - tl.w, yl0 = (sy > 0) ? tl.y0 : ny - tl.y0 - tl.h;
    const int T = (Z + tl.w + tl.h - 2 + 3) & ~3;    /* steps, in fours */
    const unsigned tag = (sm.epoch << 12) | (unsigned)(s + 1);   /* s < 2^11 */
    const int buf = s < EBUF ? s : s & 1;
    const size_t eplane = (size_t)gridDim.x * EBUF * P.rows * EW;
    if (threadIdx.x < NC) {
        /* ---- the tile's columns ---- */
        const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int lx = 8 * (wid & 1) + (lane & 7), ly = 4 * (wid >> 1) + (lane >> 3);
        const bool col = lx < tl.w && ly < tl.h;
        const bool updc = col && xl0 + lx >= lox && yl0 + ly >= loy;
        const int px = (sx > 0) ? lx : max(tl.w - 1 - lx, 0), py = (sy > 0) ? ly : max(tl.h - 1 - ly, 0);
        /* cells: x upwind / downwind, y upwind / downwind (the tile's copy is clamped to the grid) */
        const int cxU = (sx > 0) ? px : px + 1, cxD = (sx > 0) ? px + 1 : px;
        const int cyU = (sy > 0) ? py : py + 1, cyD = (sy > 0) ? py + 1 : py;
        const R HUGEV = (R)FK_HUGE;
        const R eps_r = (R)sm.src.eps_t;
        const bool ex = lx == tl.w - 1 && col, ey = ly == tl.h - 1 && col;
        unsigned long long *erow = P.edge + ((size_t)tl.tile * EBUF + buf) * P.rows * EW;   /* row of step t */
        unsigned long long *const ex0 = erow + ly, *const ey0 = erow + TY + lx;
        ptrdiff_t eoff = 0;
        int j = -lx - ly;
        const unsigned Zcol = col ? Z : 0, Zupd = updc ? Z - 1 : 0;   /* positions of the column, updated ones */
        const int iz0 = (sz > 0) ? loz - 1 : nz - loz;
        const int iz1 = iz0 + sz * j;
        /* shared-memory addresses of the item's time and z-downwind cells: a
         * column's cell k is entry k + 1, its ends repeated, so the cell is
         * entry z + 1 ascending and z descending.  Idle lanes read what is there. */
        const int dz = sz * (int)sizeof(R), cz1 = iz1 + (sz > 0);
        unsigned aT = (unsigned)__cvta_generic_to_shared(F + (py * TX + px) * zpf) + iz1 * (int)sizeof(R);
        unsigned aUU = (unsigned)__cvta_generic_to_shared(S + (cyU * (TX + 1) + cxU) * zps) + cz1 * (int)sizeof(R);
        unsigned aUD = (unsigned)__cvta_generic_to_shared(S + (cyD * (TX + 1) + cxU) * zps) + cz1 * (int)sizeof(R);
        unsigned aDU = (unsigned)__cvta_generic_to_shared(S + (cyU * (TX + 1) + cxD) * zps) + cz1 * (int)sizeof(R);
        unsigned aDD = (unsigned)__cvta_generic_to_shared(S + (cyD * (TX + 1) + cxD) * zps) + cz1 * (int)sizeof(R);
        R told = ld_shared(aT, R()), duu = ld_shared(aUU, R()), dud = ld_shared(aUD, R()), ddu = ld_shared(aDU, R()),
          ddd = ld_shared(aDD, R());                              /* this step's item */
        R zuu = 0, zud = 0, zdu = 0, zdd = 0;                     /* z-upwind cells: the item's before */
        R tv = HUGEV, tev = HUGEV, tnv = HUGEV, tnve = HUGEV;
        __syncthreads();                                          /* the border's first entries */
        for (int t0 = 0; t0 < T; t0 += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const R te = sm.plane[(u + 3) & 3][ly + 1][lx];
                const R tn = sm.plane[(u + 3) & 3][ly][lx + 1];
                const R ten = sm.plane[(u + 2) & 3][ly][lx];
                const bool valid = (unsigned)j < Zcol, upd = (unsigned)(j - 1) < Zupd;
                const R s4 = rmin(zuu, zud), s5 = rmin(zuu, zdu), s6 = rmin(zuu, duu);
                const R s1 = rmin(s4, rmin(zdu, zdd));
                const R s2 = rmin(s4, rmin(duu, dud));
                const R s3 = rmin(s5, rmin(duu, ddu));
                const R s7 = zuu;
                R r;
                bool cold = false;
                if constexpr (sizeof(R) == 4)
                    r = fk3::noinit_v<float>(mesh, tv, te, tn, tev, ten, tnv, tnve, s1, s2, s3, s4, s5, s6, s7, told);
                else
                    r = cart64<INIT>(mesh, tv, te, tn, tev, ten, tnv, tnve, s1, s2, s3, s4, s5, s6, s7, told, cold);
                /* the switch compares in the field's precision, as in the slab schedule */
                const bool near = INIT && !(rmin(rmin(tv, te), tn) > eps_r);
                if ((INIT || sizeof(R) == 8) && upd && (near || cold)) {
                    if (near) {
                        const int x = tl.x0 + px, y = tl.y0 + py;
                        r = (R)near3(sm.src, sm.mesh64, (double)tv, (double)te, (double)tn, (double)tev, (double)ten,
                                     (double)tnv, (double)tnve, (double)told, (double)s1, (double)s2, (double)s3,
                                     (double)s4, (double)s5, (double)s6, (double)s7, iz0 + sz * j + 1, x + 1, y + 1, sz,
                                     sx, sy);
                    } else if constexpr (sizeof(R) == 8) {
                        r = cart64_any(INIT, sm.mesh64, tv, te, tn, tev, ten, tnv, tnve, s1, s2, s3, s4, s5, s6, s7,
                                       told);
                    }
                }
                const R result = upd ? r : valid ? told : HUGEV;
                sm.plane[u][ly + 1][lx + 1] = result;
                st_shared_if(upd, aT, result);
                Word<R>::store(valid && ex, ex0 + eoff, eplane, tag, result);
                Word<R>::store(valid && ey, ey0 + eoff, eplane, tag, result);
                eoff += EW;
                if (CONV) {
                    const double d = upd ? (double)told - (double)result : 0.0;   /* times only decrease */
                    dmax = d > dmax ? d : dmax;
                }
                zuu = duu; zud = dud; zdu = ddu; zdd = ddd;
                tv = result;
                tev = te;
                tnv = tn;
                tnve = ten;
                ++j;
                aT += dz; aUU += dz; aUD += dz; aDU += dz; aDD += dz;
                told = ld_shared(aT, R());
                duu = ld_shared(aUU, R());
                dud = ld_shared(aUD, R());
                ddu = ld_shared(aDU, R());
                ddd = ld_shared(aDD, R());
                __syncthreads();
            }
        }
    } else {
        /* ---- the edges: lane c < TX the row above column c, TX + c the column left of row c, 24 the corner ---- */
        const int c = threadIdx.x - NC;
        const int vx = c < TX ? c : -1, vy = c < TX ? -1 : c < TX + TY ? c - TX : -1;
        /* a tile without updates in this sweep (initialisation: before the
         * source's box) reads no edge, and so starts at once */
        const bool idle = INIT && (xl0 + tl.w - 1 < lox || yl0 + tl.h - 1 < loy);
        const int ux = vx < 0 ? tl.bx - sx : tl.bx, uy = vy < 0 ? tl.by - sy : tl.by;   /* the upwind tile */
        const bool has = c <= TX + TY && !idle && vx < tl.w && vy < tl.h && ux >= 0 && ux < tl.ntx && uy >= 0 &&
                         uy < tl.nty;
        /* words follow the producer's steps: row h + (its extents) holds what step h needs */
        const int uw = vx < 0 ? min(TX, nx - TX * max(ux, 0)) : 0, uh = vy < 0 ? min(TY, ny - TY * max(uy, 0)) : 0;
        const int word = vx < 0 ? (vy < 0 ? uh - 1 : vy) : TY + vx;
        const unsigned long long *next =      /* the next word to load: step -2's */
            P.edge + ((size_t)(has ? tl.work0 + uy * tl.ntx + ux : 0) * EBUF + buf) * P.rows * EW + (has ? word : 0) +
            (ptrdiff_t)(uw + uh - 2) * EW;
        const unsigned Zw = has ? Z : 0;
        int j = -2 - (vx + vy);               /* position of the step's entry */
        R *const dst = &sm.plane[0][vy + 1][vx + 1];
        const bool writes = c <= TX + TY;
        Word<R> q[AHEAD];
        bool dead = false;
        /* a step's entry, its word loaded AHEAD steps before (in `slot`) */
        auto step = [&](int slot) {
            const bool want = (unsigned)j < Zw;
            if (!dead && !__all_sync(0xffffffffu, !want || q[slot].ok(tag))) {
                long long it = 0;
                do {
                    /* by vote: a lane that gave up alone would be missing in the next one */
                    if (++it > P.spin_limit ||
                        ((it & 63) == 0 && __any_sync(0xffffffffu, *((volatile int *)P.error) != 0))) {
                        if (c == 0) {
                            atomicCAS(P.error, 0, 4000);
                            sm.dead = 1;
                        }
                        dead = true;
                        break;
                    }
                    /* poll every word in flight: the later ones were loaded as early */
#pragma unroll
                    for (int k = 0; k < AHEAD; ++k) {
                        const int d = (k - slot) & 3;
                        if ((unsigned)(j + d) < Zw && !q[k].ok(tag)) q[k].load(next + (ptrdiff_t)(d - AHEAD) * EW, eplane);
                    }
                } while (!__all_sync(0xffffffffu, !want || q[slot].ok(tag)));
            }
            if (writes) dst[slot * ((TY + 1) * PW)] = want && !dead ? q[slot].value() : (R)FK_HUGE;
            if ((unsigned)(j + AHEAD) < Zw) q[slot].load(next, eplane);
            /* a word that had not come two steps after its load is loaded again:
             * the blocks may follow one another more closely than AHEAD steps */
            Word<R> &mid = q[(slot + 2) & 3];
            if ((unsigned)(j + 2) < Zw && !mid.ok(tag)) mid.load(next - 2 * EW, eplane);
            next += EW;
            ++j;
        };
        static_assert(AHEAD == 4, "slots follow the step modulo 4");
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
            if ((unsigned)(j + k) < Zw) q[(k + 2) & 3].load(next, eplane);
            next += EW;
        }
        step(2);
        step(3);
        __syncthreads();
        for (int t0 = 0; t0 < T; t0 += 4) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                step(u);
                __syncthreads();
            }
        }
    }
}

static __global__ void epoch_kernel(unsigned *epoch) { ++*epoch; }

/* Registers before resident tiles: FP64 with 255 takes 78 us a sweep on 41 x
 * 53 x 47, with 168 (two blocks to an SM) 89, its initialisation 0.7 and 1.0 ms. */
template <typename R, bool CONV>
__global__ void __launch_bounds__(NT, sizeof(R) == 4 ? 2 : 1) tile_kernel(Params P)
{
    extern __shared__ __align__(16) unsigned char tile_smem[];
    __shared__ Smem<R> sm;
    const int2 me = P.tiles[blockIdx.x];
    const fk_work3d_t w = P.work[me.x];
    const fk_grid3d_t g = P.grids[w.grid];
    Tile tl;
    tl.bx = me.y & 0xffff;
    tl.by = me.y >> 16;
    tl.ntx = (g.nx + TX - 1) / TX;
    tl.nty = (g.ny + TY - 1) / TY;
    tl.x0 = TX * tl.bx;
    tl.y0 = TY * tl.by;
    tl.w = min(TX, g.nx - tl.x0);
    tl.h = min(TY, g.ny - tl.y0);
    tl.tile = blockIdx.x;
    tl.work0 = P.tile0[me.x] - P.tile_base;
    const int zpf = pitch5(g.nz), zps = pitch5(g.nz + 1);
    R *F = reinterpret_cast<R *>(tile_smem) + GUARD;
    R *S = F + NC * zpf;
    R *tt = reinterpret_cast<R *>(w.tt);
    const R *slow = reinterpret_cast<const R *>(g.slow);
    const int tid = threadIdx.x, wid = tid >> 5, lane = tid & 31;
    for (int c = wid; c < NC; c += NT / 32) {
        const int x = tl.x0 + c % TX, y = tl.y0 + c / TX;
        if (c % TX < tl.w && c / TX < tl.h)
            for (int z = lane; z < g.nz; z += 32) F[c * zpf + z] = tt[((size_t)y * g.nx + x) * g.zp + z];
    }
    for (int c = wid; c < (TX + 1) * (TY + 1); c += NT / 32) {
        const int cx = min(max(tl.x0 - 1 + c % (TX + 1), 0), g.nx - 2), cy = min(max(tl.y0 - 1 + c / (TX + 1), 0), g.ny - 2);
        for (int z = lane; z <= g.nz; z += 32)
            S[c * zps + z] = slow[((size_t)cy * (g.nx - 1) + cx) * g.zcp + min(max(z - 1, 0), g.nz - 2)];
    }
    if (tid == 0) {
        fk3tw::tw_setup_src(sm.src, w, g, P.eps);
        fk3::make_mesh<double>(sm.mesh64, g.dz, g.dx, g.dy);
        sm.epoch = *P.epoch;
        sm.dead = 0;
        sm.stop = 0;
    }
    Mesh<R> mesh;
    fk3::make_mesh<R>(mesh, g.dz, g.dx, g.dy);
    __syncthreads();
    double dmax = 0.0;
    for (int s = 0; s < 8; ++s) {
        tile_sweep<R, true, CONV>(P, sm, F, S, g, tl, mesh, s, dmax);
        if (__syncthreads_or(sm.dead)) return;     /* all threads or none: the next sweep may set it again */
    }
    for (int pass = 0; pass < P.npass; ++pass) {
        dmax = 0.0;
        for (int s = 8 + 8 * pass; s < 16 + 8 * pass; ++s) {
            tile_sweep<R, false, CONV>(P, sm, F, S, g, tl, mesh, s, dmax);
            if (__syncthreads_or(sm.dead)) return;
        }
        if (CONV) {
            for (int o = 16; o > 0; o >>= 1) {
                const double v = __shfl_xor_sync(0xffffffffu, dmax, o);
                dmax = v > dmax ? v : dmax;
            }
            if (wid < 4 && lane == 0) sm.max[wid] = dmax;
            __syncthreads();
            if (tid == 0) {
                /* the pass's largest change over the work item's tiles decides for all of them */
                double m = 0.0;
                for (int k = 0; k < 4; ++k) m = sm.max[k] > m ? sm.max[k] : m;
                unsigned long long *rp = P.resid + (size_t)me.x * P.npass + pass;
                int *cp = P.pass_tiles + (size_t)me.x * P.npass + pass;
                atomicMax(rp, (unsigned long long)__double_as_longlong(m));
                __threadfence();
                atomicAdd(cp, 1);
                long long it = 0;
                while (fk3tw::ld_acquire(cp) < tl.ntx * tl.nty) {
                    if (++it > P.spin_limit || ((it & 63) == 0 && *((volatile int *)P.error) != 0)) {
                        atomicCAS(P.error, 0, 4001);
                        sm.dead = 1;
                        break;
                    }
                }
                const double r = __longlong_as_double((long long)atomicAdd(rp, 0ull));
                if (r <= P.conv_tol) {
                    sm.stop = 1;
                    atomicMin(P.conv_pass + me.x, pass);
                }
            }
            if (__syncthreads_or(sm.dead)) return;
            if (sm.stop) break;
        }
    }
    for (int c = wid; c < NC; c += NT / 32) {
        const int x = tl.x0 + c % TX, y = tl.y0 + c / TX;
        if (c % TX < tl.w && c / TX < tl.h)
            for (int z = lane; z < g.nz; z += 32) tt[((size_t)y * g.nx + x) * g.zp + z] = F[c * zpf + z];
    }
}

/* Tiles of a launch: as many as fit the chip at once, 0 if none.  The kernel's
 * shared-memory limit is the device's, the same for all calls: solvers, batches
 * and their captured graphs share the kernel. */
template <typename R, bool CONV>
int tile_capacity(int nz)
{
    int dev = 0, nsm = 0, per = 0, most = 0;
    const size_t smem = tile_bytes<R>(nz);
    cudaFuncAttributes fa;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (cudaFuncGetAttributes(&fa, tile_kernel<R, CONV>) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    const int limit = most - (int)fa.sharedSizeBytes;
    if (limit < 0 || smem > (size_t)limit) return 0;
    if (cudaFuncSetAttribute(tile_kernel<R, CONV>, cudaFuncAttributeMaxDynamicSharedMemorySize, limit) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, tile_kernel<R, CONV>, NT, smem) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    return nsm * per;
}

template <typename R, bool CONV>
int launch_tiles(const fk_grid3d_t *grids, const fk_work3d_t *work, int nwork, const fk_slabs3d_t *pl, double eps,
                 double conv_tol, int npass, cudaStream_t st)
{
    const int cap = tile_capacity<R, CONV>(pl->max_nz);
    Params P;
    P.grids = grids;
    P.work = work;
    P.tile0 = pl->tile0;
    P.edge = pl->tile_edge;
    P.epoch = pl->tile_epoch;
    P.rows = pl->max_nz + TX + TY;
    P.error = pl->error;
    P.resid = pl->resid;
    P.pass_tiles = pl->pass_slabs;
    P.conv_pass = pl->conv_pass;
    P.npass = npass;
    P.eps = eps;
    P.conv_tol = conv_tol;
    P.spin_limit = pl->spin_limit;
    const size_t smem = tile_bytes<R>(pl->max_nz);
    for (int w0 = 0; w0 < nwork;) {
        int w1 = w0;
        while (w1 < nwork && pl->work_tiles[w1 + 1] - pl->work_tiles[w0] <= cap) ++w1;
        if (w1 == w0) return (int)cudaErrorInvalidConfiguration;
        const int base = pl->work_tiles[w0], n = pl->work_tiles[w1] - base;
        P.tiles = reinterpret_cast<const int2 *>(pl->tiles) + base;
        P.tile_base = base;
        epoch_kernel<<<1, 1, 0, st>>>(pl->tile_epoch);
        void *args[] = {&P};
        const cudaError_t e = cudaLaunchCooperativeKernel((const void *)tile_kernel<R, CONV>, dim3(n), dim3(NT), args, smem, st);
        if (e != cudaSuccess) return (int)e;
        w0 = w1;
    }
    return 0;
}

} // namespace fk3tl

/* Tiles of a grid, and how many of max_nz positions a launch holds. */
extern "C" int fk3d_tiles(int nx, int ny)
{
    if ((long long)(nx + 15) / 16 > 32767 || (ny + 7) / 8 > 32767) return 0x7fffffff;
    return (nx + fk3tl::TX - 1) / fk3tl::TX * ((ny + fk3tl::TY - 1) / fk3tl::TY);
}

extern "C" int fk3d_tile_capacity(int precision, int max_nz, int converge)
{
    using namespace fk3tl;
    if (precision == 4) return converge ? tile_capacity<float, true>(max_nz) : tile_capacity<float, false>(max_nz);
    return converge ? tile_capacity<double, true>(max_nz) : tile_capacity<double, false>(max_nz);
}

extern "C" size_t fk3d_tile_edge_bytes(int precision, int ntile, int max_nz)
{
    return (size_t)ntile * fk3tl::EBUF * (max_nz + fk3tl::TX + fk3tl::TY) * fk3tl::EW * 8 * (precision / 4);
}

/* The sweeps of a solve (fields initialised, bookkeeping cleared). */
extern "C" int fk3d_sweep_tiles(int precision, const fk_grid3d_t *grids, const fk_work3d_t *work, int nwork,
                                const fk_slabs3d_t *pl, double eps, int npass, int converge, double conv_tol,
                                cudaStream_t st)
{
    using namespace fk3tl;
    if (precision == 4)
        return converge ? launch_tiles<float, true>(grids, work, nwork, pl, eps, conv_tol, npass, st)
                        : launch_tiles<float, false>(grids, work, nwork, pl, eps, conv_tol, npass, st);
    return converge ? launch_tiles<double, true>(grids, work, nwork, pl, eps, conv_tol, npass, st)
                    : launch_tiles<double, false>(grids, work, nwork, pl, eps, conv_tol, npass, st);
}
