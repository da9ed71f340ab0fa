// mg.cu -- the reference's Poisson solver (iterative_solver.f90 -> mg.f90 -> sors.f90) as
// ONE persistent cooperative kernel: every V-cycle, every red-black SOR sweep and every
// convergence decision runs on the device; no host round trip per sweep or per cycle.
//
// Compiled with -fmad=false: the SOR update, the residual and the restriction weights are
// rounded exactly as the Fortran expressions are written, so with the same sweep counts the
// result equals the FP64 CPU restatement bit for bit.  The L1 residual sums are reduced in a
// fixed order (per-thread, warp tree, warps, CTAs), so a solve is reproducible run to run.
//
// What bounds it: not bytes (a 513^2 level and its right-hand side are 4 MB, in L2) but the
// chain of dependent steps.  The reference decides after every sweep whether to go on, so a
// sweep run grid-wide costs three grid barriers (red, black, residual) of about 2-3 us, and a
// sweep of a coarse level by one CTA out of global memory about 10 us.  So:
//  * Levels above the CTA-0 part are swept in shared-memory tiles (temporal blocking): a CTA
//    loads a tile of u, b and the mask with a halo, runs all K sweeps of a stage there (half-
//    sweep h updates the nodes at least h + 1 nodes inside the region, so the tile ends with
//    exactly the values of grid-wide sweeps), sums each sweep's residual on the way, and
//    restricts the result into the next level's right-hand side in the same pass (or starts
//    from the prolongation of the coarser correction): one grid barrier per stage.  K is the
//    number of sweeps the stage took in the previous cycle.  The decisions are taken afterwards
//    from the K sums, which are the reference's: if it would have stopped earlier, the pass is
//    run again from its untouched input with that many sweeps; if not yet, another pass follows.
//  * Levels of at most mg_small_nodes nodes live in CTA 0's shared memory (u, b, mask) for the
//    whole solve, under the same prediction: K sweeps, then one reduction of their K sums.
//  * A sweep in shared memory is bound by its loads and by what surrounds the arithmetic: u, b
//    and the mask are kept by colour (unit stride, two wavefronts per load instead of four),
//    addressed by 32-bit shared-memory offsets with no row or column to work out, and a
//    thread's residual sums go to a slot of its own that is reduced once per stage.
// Measured (B200, warm solve to 1e-8, 4 cycles): 129^2 nodes 2.32 -> 0.64 ms, 513^2 3.05 -> 1.20 ms,
// 384 x 256 cells with periodic edges 3.43 -> 1.12 ms; 513^2 cold to the L1 1e-10 4.96 -> 1.66 ms.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include "lepic_internal.cuh"

struct MGDev {
    int nx, ny;
    double aw, an, ac;    // mg.h:11-15 (ae = aw, as = an)
    double y;             // 1 / ac (0: ac out of the range of quot())
    double *u, *u2;       // the level's two buffers: a pass reads one and writes the other
    double *b;
    const int8_t *bc;
    int tx, ty;           // the tile of the level's passes
    int seam;             // its residuals are final only after the edge rows' copy: summed in a pass of their own
    int su, sb, sm;       // levels of the CTA-0 part: offsets of u, b (doubles) and the mask (bytes)
};

struct MGP {
    MGDev L[LEPIC_MAXLEV];
    int ng, Ls;           // levels >= Ls are handled by CTA 0
    double omega, eps, alpha;
    int ncycl, pbc, nmn, mode;
    int cap;              // nodes a tile's region may hold
    double *partials;
    DevCounters *cnt;
    unsigned bar_extra;        // lepic_options::barrier_extra
};

#define MGT 512           // threads per CTA, one CTA per SM
#define MGW (MGT / 32)
#define MG_NB 2           // nodes a thread updates at a time
#define MG_KMAX 4         // sweeps per pass
#define MG_HMAX (2 * MG_KMAX + 2)
#define MG_NSUM (MG_KMAX + 2)   // a pass's sums: |r| per sweep, r^2 after the last, ||b0||^2
#define MG_NR 10          // sweeps per stage at most (but the coarsest level's in the first cycle)
#define MG_SLOTS 5120     // doubles at the start of shared memory: each thread's sum of each sweep (MG_NR MGT), a level's residual

extern __shared__ __align__(16) double smd[];

// A patch of a level in shared memory: the columns [ri0, ri0 + RW) and up to two runs of rows
// (the second where the halo wraps around a periodic edge).  The row pitch is odd and the runs
// are spaced so that i + j and the flat index q agree in parity up to a constant: a half-sweep
// is a loop over every second q, with no rows or columns to work out; the two colours of u, b and
// the mask are kept apart, so that consecutive threads read consecutive words.  What is to be done
// at a node is in its mask byte:
#define M_WALL 1     // a wall, or outside the level
#define M_IN (-1)    // updated, and its residual counts (bcnd -1 in the tile)
#define M_UPD 0      // updated (the same in the halo, and labels that the residual leaves out)
#define M_NMN (-2)   // updated with the Neumann stencil
#define M_FIX (-16)  // bcnd <= 0 but not updated (ghosts, the periodic copy, the region's rim)
struct Patch {
    int nx, ny;
    int i0, i1, j0, j1;      // the tile's updatable nodes
    int ri0, RW, RH, RP;     // RP: row pitch
    int nA, n0, a0, b0;      // local row lr is row a0 + lr for lr < nA, b0 + lr - n0 from n0, else none
    int clip0, clip1;        // rows that the level's edge cut off the halo, below and above
    int par;                 // parity of i + j at q = 0
    int wrap;                // 0: one run; 1: wrapped rows first (below row 1); 2: last; 3: every row
    int PS;                  // nodes of one colour: q is element px(q) of its array
    int uo, bo, mo;          // the arrays' offsets in shared memory (u, b in doubles, the mask in bytes)
    __device__ __forceinline__ int px(int q) const { return (q & 1) * PS + (q >> 1); }
    __device__ __forceinline__ double &u(int q) const { return smd[uo + px(q)]; }
    __device__ __forceinline__ double &b(int q) const { return smd[bo + px(q)]; }
    __device__ __forceinline__ int8_t &m(int q) const { return ((int8_t *)smd)[mo + px(q)]; }
    __device__ __forceinline__ int row_of(int lr) const { return lr < nA ? a0 + lr : (lr < n0 ? -1 : b0 + lr - n0); }
    // the local row of the tile's own run
    __device__ __forceinline__ int own(int j) const { return wrap == 2 ? j - a0 : n0 + j - b0; }
};

#define CLIP_ALL (1 << 20)   // no row of the region ever falls out of reach

__device__ __forceinline__ Patch tile_patch(const MGP &P, const MGDev &L, int tile, int H) {
    Patch g;
    const int nx = L.nx, ny = L.ny, TX = L.tx, TY = L.ty;
    const int ntx = (nx + 1 + TX - 1) / TX;
    const int tj = tile / ntx, ti = tile - tj * ntx;
    g.nx = nx; g.ny = ny;
    g.i0 = 1 + ti * TX;
    g.j0 = 1 + tj * TY;
    g.i1 = min(g.i0 + TX, nx + 2);
    g.j1 = min(g.j0 + TY, ny + 2);
    g.ri0 = max(g.i0 - H, 0);
    g.RW = min(g.i1 + H, nx + 3) - g.ri0;
    g.RP = mg_pitch(g.RW);
    g.wrap = 0; g.nA = g.n0 = 0; g.a0 = 0;
    g.b0 = max(g.j0 - H, 0);
    g.RH = min(g.j1 + H, ny + 3) - g.b0;
    g.clip0 = g.b0 - (g.j0 - H);
    g.clip1 = g.j1 + H - (g.b0 + g.RH);
    if (P.pbc) {
        const bool below = g.j0 - H < 1, above = g.j1 + H - 1 > ny;
        if (below && above) g.wrap = 3;
        else if (below) g.wrap = g.j1 + H > ny + g.j0 - H ? 3 : 1;
        else if (above) g.wrap = g.j1 + H - ny >= g.j0 - H ? 3 : 2;
        if (g.wrap) { g.b0 = 0; g.clip0 = g.clip1 = 0; }
        if (g.wrap == 3) { g.RH = ny + 3; g.clip0 = g.clip1 = CLIP_ALL; }
        else if (g.wrap == 1) {          // rows .. ny + 1, then 0 .. (row 0 follows at the parity of ny)
            g.a0 = ny + g.j0 - H; g.nA = ny + 2 - g.a0; g.n0 = g.nA + (ny & 1);
            g.RH = g.n0 + g.j1 + H;
        } else if (g.wrap == 2) {        // rows .. ny + 2, then 0 ..
            g.a0 = g.j0 - H; g.nA = ny + 3 - g.a0; g.n0 = g.nA + ((ny + 1) & 1);
            g.RH = g.n0 + g.j1 + H - ny;
        }
    }
    g.par = (g.ri0 + (g.nA ? g.a0 : g.b0)) & 1;
    g.PS = mg_plane(g.RP, g.RH);
    g.uo = MG_SLOTS;
    g.bo = MG_SLOTS + P.cap;
    g.mo = 8 * (MG_SLOTS + 2 * P.cap);
    return g;
}

// a whole level in CTA 0's shared memory
__device__ __forceinline__ Patch level_patch(const MGP &P, int l) {
    const MGDev &L = P.L[l];
    Patch g;
    g.nx = L.nx; g.ny = L.ny;
    g.i0 = 1; g.i1 = L.nx + 2; g.j0 = 1; g.j1 = L.ny + 2;
    g.ri0 = 0; g.RW = L.nx + 3; g.RP = mg_pitch(g.RW); g.RH = L.ny + 3;
    g.nA = g.n0 = 0; g.a0 = 0; g.b0 = 0;
    g.clip0 = g.clip1 = CLIP_ALL;
    g.par = 0;
    g.wrap = P.pbc ? 3 : 0;
    g.PS = mg_plane(g.RP, g.RH);
    g.uo = MG_SLOTS + L.su;
    g.bo = MG_SLOTS + L.sb;
    g.mo = 8 * MG_SLOTS + L.sm;
    return g;
}

// the mask byte of node (i, j) with boundary label bc; own: a row of the tile's own run
__device__ __forceinline__ int8_t mask_of(const Patch &g, int bc, int i, int j, bool own) {
    if (bc > 0) return M_WALL;
    if (i < 1 || i > g.nx + 1 || j < 1 || j > g.ny + 1 || (bc == 0 && j == g.ny + 1) || i == g.ri0 || i == g.ri0 + g.RW - 1)
        return M_FIX;
    if (bc == -2) return M_NMN;
    return bc == -1 && own && i >= g.i0 && i < g.i1 && j >= g.j0 && j < g.j1 ? M_IN : M_UPD;
}

// lanes per row (log2): a warp takes one, two or four rows at a time, whichever fits their width
__device__ __forceinline__ int lanes_of(int width) { return width <= 8 ? 3 : (width <= 16 ? 4 : 5); }

// t / ac, correctly rounded, for the level's fixed divisor with y = RN(1 / ac): q0 = RN(t y) is
// within 1.5 ulp, so the first correction by the exact remainder leaves a quotient within one ulp
// and the second rounds it correctly (P. Markstein, "Computation of elementary functions on the
// IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990: y correctly rounded and q within an
// ulp make q + (t - ac q) y correctly rounded).  Five dependent operations of 8 cycles against
// about 100 cycles of the general division, in the middle of every update's chain.  The
// remainders are exact while t is neither tiny nor huge; outside that range (and where the host
// found ac itself out of range: y = 0) the general division is used.
__device__ __noinline__ double quot_general(double t, double ac) { return t / ac; }
__device__ __forceinline__ double quot(double t, double ac, double y) {
    const unsigned hi = (unsigned)__double2hiint(t) & 0x7fffffffu;
    double q = t * y;
    q = __fma_rn(__fma_rn(-ac, q, t), y, q);
    q = __fma_rn(__fma_rn(-ac, q, t), y, q);
    if ((hi - 0x07c00000u >= 0x70800000u && t != 0.0) || y == 0.0) q = quot_general(t, ac);
    return q;
}

// |r| (RES) of the sweeps' last half-sweep's other colour (red), or of both colours, and r^2 of
// both, over the tile's nodes
__device__ __forceinline__ void last_residual(const Patch &g, const MGDev &L, double &acc, double &l2, int T, bool both, bool sq) {
    const double aw = L.aw, an = L.an, ac = L.ac;
    const int RP = g.RP, PS = g.PS, lo = RP, hi = (g.RH - 1) * RP;
    for (int c = 0; c < (both || sq ? 2 : 1); c++) {        // red, then black
        const int pl = (g.par ^ 1 ^ c) & 1;
        const int own = g.uo + pl * PS, nb = g.uo + (pl ^ 1) * PS + pl, bo = g.bo + pl * PS, mo = g.mo + pl * PS;
        const int up = nb + (RP - 1) / 2, dn = nb - (RP + 1) / 2, pe = (hi - pl + 1) >> 1;
        for (int p = ((lo - pl + 1) >> 1) + (int)threadIdx.x; p < pe; p += T) {
            const double r = smd[bo + p] - (aw * smd[nb + p - 1] + an * smd[up + p] + an * smd[dn + p] + aw * smd[nb + p] + ac * smd[own + p]);
            if (((const int8_t *)smd)[mo + p] != M_IN) continue;
            if (both || c == 0) acc += fabs(r);
            if (sq) l2 += r * r;
        }
    }
}

// The stencil's coefficients and one colour's arrays, held in registers through a stage
struct Coef { double aw, an, ac, y, om, omo; };
struct Plane { int own, w, n, s, b, m, pl; };   // offsets of the colour's nodes, neighbours (east is w + 1), b, mask
__device__ __forceinline__ Plane plane_of(const Patch &g, int color) {
    Plane c;
    c.pl = (g.par ^ 1 ^ color) & 1;           // red (0) is i + j odd, black (1) even
    const int nb = g.uo + (c.pl ^ 1) * g.PS + c.pl;
    c.own = g.uo + c.pl * g.PS;
    c.w = nb - 1;
    c.n = nb + (g.RP - 1) / 2;
    c.s = nb - (g.RP + 1) / 2;
    c.b = g.bo + c.pl * g.PS;
    c.m = g.mo + c.pl * g.PS;
    return c;
}

// One node's SOR update (sors.f90:80-118 / :210-248) from its loaded values; adds |r| of the
// value before (PRE) or after the update (sors.f90:338-357) to acc where it counts
struct NodeIn { double uo, uw, ue, un, us, b; int m; };
__device__ __forceinline__ NodeIn node_load(const Plane &c, int p) {
    NodeIn v;
    v.m = ((const int8_t *)smd)[c.m + p];
    v.uo = smd[c.own + p]; v.uw = smd[c.w + p]; v.ue = smd[c.w + 1 + p]; v.un = smd[c.n + p]; v.us = smd[c.s + p];
    v.b = smd[c.b + p];
    return v;
}
template <bool PRE>
__device__ __forceinline__ void node_update(const NodeIn &v, double *u, const Coef &k, double &acc) {
    if ((unsigned)(-v.m) > 4u) return;
    const double pw = k.aw * v.uw, pn = k.an * v.un, ps = k.an * v.us, pe = k.aw * v.ue;
    double t = v.b - pw - pn - ps - pe;
    if (v.m == M_NMN) t = v.b - pn - ps - 2.0 * k.aw * v.ue;
    const double unew = k.omo * v.uo + quot(k.om * t, k.ac, k.y);
    *u = unew;
    if (v.m == M_IN) acc += fabs(v.b - (pw + pn + ps + pe + k.ac * (PRE ? v.uo : unew)));
}

// Half-sweep of one colour over the flat range [lo, hi) by a team of T threads; returns the thread's
// sum of |r|
template <bool PRE>
__device__ __forceinline__ double half_sweep(const Plane &c, const Coef &k, int lo, int hi, int T) {
    double acc = 0.0;
    const int pe = (hi - c.pl + 1) >> 1;
    int p = ((lo - c.pl + 1) >> 1) + (int)threadIdx.x;
    for (; p + (MG_NB - 1) * T < pe; p += MG_NB * T) {   // MG_NB nodes at a time: their chains overlap
        NodeIn v[MG_NB];
#pragma unroll
        for (int i = 0; i < MG_NB; i++) v[i] = node_load(c, p + i * T);
#pragma unroll
        for (int i = 0; i < MG_NB; i++) node_update<PRE>(v[i], smd + c.own + p + i * T, k, acc);
    }
    if (p + T < pe) {
        const NodeIn v0 = node_load(c, p), v1 = node_load(c, p + T);
        node_update<PRE>(v0, smd + c.own + p, k, acc);
        node_update<PRE>(v1, smd + c.own + p + T, k, acc);
        p += 2 * T;
    }
    if (p < pe) node_update<PRE>(node_load(c, p), smd + c.own + p, k, acc);
    return acc;
}

// ||b - A u_D||^2 of the tile (u_D: u with the unknowns zeroed) over bcnd == -1
__device__ __forceinline__ double wall_norm(const Patch &g, const MGDev &L) {
    const double aw = L.aw, an = L.an;
    const int RP = g.RP;
    double s = 0.0;
    for (int q = RP + (int)threadIdx.x; q < (g.RH - 1) * RP; q += MGT) {
        if (g.m(q) != M_IN) continue;
        const double d = g.b(q) - ((g.m(q - 1) > 0 ? aw * g.u(q - 1) : 0.0) + (g.m(q + RP) > 0 ? an * g.u(q + RP) : 0.0) +
                                   (g.m(q - RP) > 0 ? an * g.u(q - RP) : 0.0) + (g.m(q + 1) > 0 ? aw * g.u(q + 1) : 0.0));
        s = s + d * d;
    }
    return s;
}

// sors.f90:185-200 periodic ghost rows: row 0 is row ny, row ny + 1 is row 1
__device__ __forceinline__ void pbc_rows(const Patch &g, int T) {
    if (!g.wrap) return;
    const int ny = g.ny, RP = g.RP;
    const int hi = g.wrap == 3 ? 0 : g.a0, lo = g.wrap == 3 ? 0 : g.n0;   // local rows: j - hi near ny, lo + j near 0
    for (int k = threadIdx.x; k < g.RW; k += T) {
        if (g.m(k + (lo + 1) * RP) <= 0) g.u(k + lo * RP) = g.u(k + (ny - hi) * RP);
        if (g.m(k + (ny + 1 - hi) * RP) <= 0) g.u(k + (ny + 1 - hi) * RP) = g.u(k + (lo + 1) * RP);
    }
}

// mg.f90:512-547 at local node q, column ir
__device__ __forceinline__ double getres(const Patch &g, const MGDev &L, int q, int ir, int flag) {
    double aw = L.aw, ae = L.aw, an = L.an, as = L.an;
    const double ac = L.ac;
    double uij = g.u(q), un = g.u(q + g.RP), us = g.u(q - g.RP), ue = g.u(q + 1), uw = g.u(q - 1);
    if (ir == 1 && flag == 1) {
        uw = 0.0;
        aw = 0;
        ae = 2.0 * ae;
    }
    return g.b(q) - (aw * uw + ae * ue + an * un + as * us + ac * uij);
}

// The fine residual on the tile and one node around it, to smd[ro + px(q)] (ro = g.bo: in place of
// b, when the sweeps on it are done)
__device__ __forceinline__ void residual_to(const Patch &g, const MGDev &L, int nmn, int ro) {
    const int RP = g.RP;
    const int c0 = max(g.i0 - 1, 1), c1 = min(g.i1 + 1, g.nx + 2);
    const int lg = lanes_of(c1 - c0), lpr = 1 << lg;
    const int lane = threadIdx.x & (lpr - 1), sub = threadIdx.x >> lg, nsub = MGT >> lg;
    // r_pbc reads row ny: the wrapped run's last but one row, or any row when all are here
    const int l0 = g.wrap == 3 ? 1 : (g.wrap == 1 ? g.ny - g.a0 : g.own(max(g.j0 - 1, 1)));
    const int l1 = g.wrap == 3 ? g.ny + 2 : g.own(min(g.j1, g.ny + 1)) + 1;
#pragma unroll 2
    for (int lr = l0 + sub; lr < l1; lr += nsub) {
        const int j = g.row_of(lr);
        if (j < 1 || (g.wrap == 1 && lr < g.n0 && j != g.ny)) continue;
        for (int i = c0 + lane; i < c1; i += lpr) {
            const int q = lr * RP + i - g.ri0;
            if (g.m(q) <= 0 || (g.wrap && j == g.ny)) smd[ro + g.px(q)] = getres(g, L, q, i, nmn);
        }
    }
}

// mg.f90:235-509 on one rank: full-weighting restriction of the fine residual (held at ro) at
// the coarse nodes whose fine centre lies in the tile; put(i, j, value) stores it (the coarse
// mask is the precomputed injection, its value read by mask(i, j))
template <class Mask, class Put>
__device__ __forceinline__ void restriction(const Patch &g, int pbc, int ro, Mask mask, Put put) {
    const int nx = g.nx, ny = g.ny, RP = g.RP;
    const int ic0 = (g.i0 + 2) / 2, ic1 = g.i1 / 2 + 1, jc0 = (g.j0 + 2) / 2, jc1 = g.j1 / 2 + 1;
    const int lg = lanes_of(ic1 - ic0), lpr = 1 << lg;
    const int lane = threadIdx.x & (lpr - 1), sub = threadIdx.x >> lg, nsub = MGT >> lg;
    const int lny = g.wrap == 3 ? ny : ny - g.a0;    // local row of ny (periodic)
    // r_pbc(x) of mg.f90:298-311 (zero where the reference leaves it unset)
    auto rpbc = [&](int x) {
        const int t = (lny + 1) * RP + x - g.ri0;
        bool set;
        if (x & 1) set = g.m(t) <= 0;
        else set = (x - 1 >= 1 && g.m(t - 1) <= 0) || (x + 1 <= nx + 1 && g.m(t + 1) <= 0);
        return set ? smd[ro + g.px(t - RP)] : 0.0;
    };
    for (int j = jc0 + sub; j < jc1; j += nsub)
        for (int i = ic0 + lane; i < ic1; i += lpr) {
            const int ir = 2 * i - 1, jr = 2 * j - 1;
            double out = 0.0;
            if (mask(i, j) <= 0) {
                const int q = g.own(jr) * RP + ir - g.ri0;
                auto r = [&](int d) { return smd[ro + g.px(q + d)]; };
                auto m = [&](int d) { return (int)g.m(q + d); };
                double r1 = 0, r2 = 0, r3 = 0, r4 = 0, r5 = 0, r6 = 0, r7 = 0, r8 = 0;
                const double r9 = r(0);
                if (ir != nx + 1 && jr != ny + 1)
                    if (m(1 + RP) <= 0) r1 = r(1 + RP);
                if (ir != nx + 1)
                    if (m(1) <= 0) r2 = r(1);
                if (m(1 - RP) <= 0) {
                    if (ir != nx + 1 && jr != 1) r3 = r(1 - RP);
                    else if (jr == 1) r3 = pbc && ir <= nx ? rpbc(ir + 1) : 0.0;   // zero past a free right column too
                }
                if (m(-RP) <= 0) {
                    if (jr != 1) r4 = r(-RP);
                    else r4 = pbc ? rpbc(ir) : 0.0;
                }
                if (m(-1 - RP) <= 0 && ir != 1) {
                    if (jr != 1) r5 = r(-1 - RP);
                    else r5 = pbc ? rpbc(ir - 1) : 0.0;
                }
                if (m(-1) <= 0)
                    if (ir != 1) r6 = r(-1);
                if (m(-1 + RP) <= 0)
                    if (ir != 1 && jr != ny + 1) r7 = r(-1 + RP);
                if (m(RP) <= 0)
                    if (jr != ny + 1) r8 = r(RP);
                out = (4.0 * r9 + 2.0 * (r2 + r4 + r6 + r8) + r1 + r3 + r5 + r7) / 16.0;
            }
            put(i, j, out);
        }
}

// mg.f90:549-616 at fine node (i, j), 0 <= i <= nx + 1, 0 <= j <= ny + 1: u plus the coarse
// correction e(index), rows of W2 (each fine node has one coarse node whose stencil holds it)
template <class E>
__device__ __forceinline__ double prolonged(double u, E e, int W2, int i, int j) {
    const int p = (i + 2) / 2 + ((j + 2) / 2) * W2;
    const double r1 = e(p);
    if (i & 1) {
        if (j & 1) return u + r1;
        return u + (r1 + e(p - W2)) / 2.0;
    }
    if (j & 1) return u + (r1 + e(p - 1)) / 2.0;
    return u + (r1 + e(p - W2) + e(p - 1 - W2) + e(p - 1)) / 4.0;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = v + __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// one double global -> shared without a register round trip
__device__ __forceinline__ void cp_async8(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

struct MGShared {
    Patch g;                        // the tile being worked on
    Patch lev[LEPIC_MAXLEV];        // the levels of the CTA-0 part
    double tot[MG_NR];              // the sums of the last pass or stage
    double red[MGW], res;           // CTA 0's sums and last residual
    int pred[2][LEPIC_MAXLEV];      // sweeps a stage took last time, down and up
    int iter[LEPIC_MAXLEV];
};

#define SRC_ZERO 0        // a correction: starts from zeros
#define SRC_U 1           // the level's current buffer
#define SRC_UP 2          // ... plus the prolongation of the next level's

__device__ __forceinline__ double *buf_of(const MGDev &L, int which) { return which ? L.u2 : L.u; }

// the barrier of the CTA's first T threads (T a multiple of 32)
__device__ __forceinline__ void team_sync(int T) {
    if (T == 32) __syncwarp();
    else asm volatile("bar.sync 1, %0;" :: "r"(T) : "memory");
}

// K sweeps of a patch by a team of T threads; each thread puts its sum of sweep k's |r| into slot k,
// and of r^2 after the last sweep into slot MG_KMAX with l2 (add: on top of what the slot holds).  A
// black half-sweep sums the residuals of its own nodes (their red neighbours are final), the
// next red one those of the red nodes before it updates them.  Rows within h + 1 of the region's
// cut edge hold values that can no longer reach the tile in half-sweep h and are left out
// (columns there are updated like the rest; what they hold reaches no further either).
__device__ __forceinline__ void sweeps(const MGP &P, const Patch &g, const MGDev &L, int K, int T, bool l2, bool add) {
    double *const slot = smd + threadIdx.x;
    const bool pbc = P.pbc != 0, seam = L.seam != 0;
    const Coef k{L.aw, L.an, L.ac, L.y, P.omega, 1.0 - P.omega};
    const Plane red = plane_of(g, 0), black = plane_of(g, 1);
    const int RP = g.RP, RH = g.RH, c0 = g.clip0, c1 = g.clip1;
    double a0 = 0.0, unused = 0.0;
    for (int s = 0; s < K; s++) {
        double a = half_sweep<true>(red, k, max(1, 2 * s + 1 - c0) * RP, (RH - max(1, 2 * s + 1 - c1)) * RP, T);
        if (s) {
            if (!seam) a0 += a;
            slot[(s - 1) * MGT] = add ? slot[(s - 1) * MGT] + a0 : a0;
        }
        team_sync(T);
        if (pbc) { pbc_rows(g, T); team_sync(T); }
        a0 = half_sweep<false>(black, k, max(1, 2 * s + 2 - c0) * RP, (RH - max(1, 2 * s + 2 - c1)) * RP, T);
        team_sync(T);
        if (pbc) { pbc_rows(g, T); team_sync(T); }
        if (seam) {
            a0 = 0.0;
            last_residual(g, L, a0, unused, T, true, false);
            team_sync(T);
        }
    }
    double q2 = 0.0;
    if (l2) last_residual(g, L, seam ? unused : a0, q2, T, false, true);
    else if (!seam) last_residual(g, L, a0, q2, T, false, false);
    slot[(K - 1) * MGT] = add ? slot[(K - 1) * MGT] + a0 : a0;
    if (l2) slot[MG_KMAX * MGT] = add ? slot[MG_KMAX * MGT] + q2 : q2;
}

// slot k summed over the team's threads in a fixed order, by one warp
__device__ __forceinline__ double slot_sum(int k, int T) {
    double a = 0.0;
    for (int t = threadIdx.x & 31; t < T; t += 32) a = a + smd[k * MGT + t];
    return warp_sum(a);
}

// The reference's decisions (sors.f90:360-400) from the K sums S.tot of sweeps done + 1 .. done + K:
// returns how many of them it takes (K: it goes on, unless stop); res_s: the sum before them (0:
// none).  Lane k decides sweep k.
__device__ __forceinline__ int decide(const MGP &P, const MGShared &S, int K, int done, int nr, int dig, double &res, double &res_s,
                                      bool &stop) {
    const int lane = threadIdx.x & 31;
    const double cur = lane < K ? S.tot[lane] : 0.0;
    double prev = __shfl_up_sync(0xffffffffu, cur, 1);
    if (lane == 0) prev = res_s;
    bool st = lane < K;
    if (dig == 0) st = st && cur <= P.eps * P.alpha;
    else st = st && prev > 0.0 && (cur / prev) <= 0.6;
    const unsigned hit = __ballot_sync(0xffffffffu, st);
    const int q = hit ? __ffs(hit) : K;
    stop = hit != 0 || done + K == nr;
    res = __shfl_sync(0xffffffffu, cur, q - 1);
    res_s = res;
    return q;
}

// One pass over level l: K sweeps of every tile from buffer `cur` into the other one.  Sums of
// the pass into the slots (summed over this CTA's tiles).
__device__ __forceinline__ void tile_pass(const MGP &P, MGShared &S, int l, int cur, int src, int ccur, int K, bool restr, bool l2,
                          bool bb) {
    const MGDev &L = P.L[l];
    const Patch &g = S.g;              // in shared memory: read where needed, no registers held
    const int nx = L.nx, ny = L.ny, W = nx + 3;
    const double *uin = buf_of(L, cur);
    double *uout = buf_of(L, cur ^ 1);
    for (int k = 0; k < MG_NSUM; k++) smd[k * MGT + threadIdx.x] = 0.0;
    const int ntiles = ((nx + 1 + L.tx - 1) / L.tx) * ((ny + 1 + L.ty - 1) / L.ty);
    const int first = P.Ls < P.ng ? 1 : 0;       // CTA 0 keeps its shared memory for the coarse levels
    const int H = 2 * K + (restr ? 2 : 1);
    for (int tile = (int)blockIdx.x - first; tile >= 0 && tile < ntiles; tile += (int)gridDim.x - first) {
        if (threadIdx.x == 0) S.g = tile_patch(P, L, tile, H);
        __syncthreads();
        const int lg = lanes_of(g.RP), lpr = 1 << lg;
        const int ln = threadIdx.x & (lpr - 1), sub = threadIdx.x >> lg, nsub = MGT >> lg;
        for (int lr = sub; lr < g.RH; lr += nsub) {
            const int j = g.row_of(lr);
            const bool jb = j >= 1 && j <= ny + 1;
            for (int k = ln; k < g.RW; k += lpr) {
                const int i = g.ri0 + k, q = lr * g.RP + k;
                if (jb && i >= 1 && i <= nx + 1)
                    cp_async8(&g.b(q), L.b + (i - 1) + (long long)(j - 1) * (nx + 1));
                else
                    g.b(q) = 0.0;
                if (src == SRC_ZERO || j < 0) g.u(q) = 0.0;
                else cp_async8(&g.u(q), uin + i + (long long)j * W);
            }
        }
        // the mask bytes of four rows at a time, so that their loads overlap
        for (int lr0 = sub; lr0 < g.RH; lr0 += 4 * nsub)
            for (int k = ln; k < g.RP; k += lpr) {
                int bc[4];
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const int lr = lr0 + v * nsub;
                    const int j = lr < g.RH ? g.row_of(lr) : -1;
                    bc[v] = j >= 0 && k < g.RW ? (int)__ldg(L.bc + g.ri0 + k + (long long)j * W) : 1;
                }
#pragma unroll
                for (int v = 0; v < 4; v++) {
                    const int lr = lr0 + v * nsub;
                    if (lr < g.RH)
                        g.m(lr * g.RP + k) = mask_of(g, bc[v], g.ri0 + k, g.row_of(lr), g.wrap == 2 ? lr < g.nA : lr >= g.n0);
                }
            }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (src == SRC_UP) {
            const MGDev &C = P.L[l + 1];
            const double *e = buf_of(C, ccur);
            const int W2 = C.nx + 3;
#pragma unroll 2
            for (int lr = sub; lr < g.RH; lr += nsub) {
                const int j = g.row_of(lr);
                if (j < 0 || j > ny + 1) continue;
                for (int k = ln; k < g.RW; k += lpr) {
                    const int i = g.ri0 + k, q = lr * g.RP + k;
                    if (i <= nx + 1 && g.m(q) <= 0) g.u(q) = prolonged(g.u(q), [&](int t) { return e[t]; }, W2, i, j);
                }
            }
            __syncthreads();
        }
        if (bb) smd[(MG_KMAX + 1) * MGT + threadIdx.x] += wall_norm(g, L);
        sweeps(P, g, L, K, MGT, l2, true);
        // the tile, and for a tile on the border the ghost nodes beside it: the tiles together
        // write every node of the level exactly once
        {
            const int wi0 = g.i0 == 1 ? 0 : g.i0, wj0 = g.j0 == 1 ? 0 : g.j0;
            const int wi1 = g.i1 == nx + 2 ? nx + 3 : g.i1, wj1 = g.j1 == ny + 2 ? ny + 3 : g.j1;
            for (int j = wj0 + sub; j < wj1; j += nsub)
                for (int i = wi0 + ln; i < wi1; i += lpr)
                    uout[i + (long long)j * W] = g.u(g.own(j) * g.RP + i - g.ri0);
        }
        if (restr) {
            const MGDev &C = P.L[l + 1];
            __syncthreads();           // the residual sums have read b
            residual_to(g, L, P.nmn, g.bo);
            __syncthreads();
            restriction(g, P.pbc, g.bo, [&](int i, int j) { return (int)__ldg(C.bc + i + (long long)j * (C.nx + 3)); },
                        [&](int i, int j, double v) { C.b[(i - 1) + (long long)(j - 1) * (C.nx + 1)] = v; });
        }
        __syncthreads();
    }
}

// every CTA's slots summed in a fixed order into S.tot, behind the grid barrier that also ends
// the pass; the sums alternate between the halves of `partials`, so that a CTA that runs ahead
// writes none of the slots still being read
__device__ bool pass_sums(const MGP &P, MGShared &S, unsigned *phase) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    double *part = P.partials + (*phase & 1) * MG_NSUM * gridDim.x;
    *phase += 1;
    if (warp < MG_NSUM) {
        const double a = slot_sum(warp, MGT);
        if (lane == 0) part[warp * gridDim.x + blockIdx.x] = a;
    }
    if (!grid_barrier(P.cnt, gridDim.x + P.bar_extra)) return false;
    if (warp < MG_NSUM) {
        double a = 0.0;
        for (int i = lane; i < (int)gridDim.x; i += 32) a = a + __ldcg(part + warp * gridDim.x + i);
        a = warp_sum(a);
        if (lane == 0) S.tot[warp] = a;
    }
    __syncthreads();
    return true;
}

// sors.f90:1-435 on one rank for a level of the tile passes; false when a barrier failed.  dir: 0
// down, 1 up (where the predicted sweep count is kept)
__device__ bool sor_big(const MGP &P, MGShared &S, int l, int kmg, int dig, int dir, int src, bool restr, bool l2,
                        bool bb, unsigned &curs, unsigned *phase, double *res_out, double *bb_out) {
    double res = 0.0, res_s = 0.0;
    const int nr = kmg == 1 && dig == 0 ? 1000000 : MG_NR;
    const int want = S.pred[dir][l];
    int done = 0;
    bool stop = false;
    while (!stop) {
        // more than MG_KMAX sweeps are split evenly; past the prediction two, then MG_KMAX
        int K = done ? MG_KMAX : 2;
        if (done < want) {
            const int left = want - done, parts = (left + MG_KMAX - 1) / MG_KMAX;
            K = (left + parts - 1) / parts;
        }
        K = min(K, nr - done);
        const int cur = (curs >> l) & 1, ccur = (curs >> (l + 1)) & 1;
        tile_pass(P, S, l, cur, src, ccur, K, restr, l2, bb);
        if (!pass_sums(P, S, phase)) return false;
        if (bb) *bb_out = S.tot[MG_KMAX + 1];
        bb = false;
        const int q = decide(P, S, K, done, nr, dig, res, res_s, stop);
        if (q < K) {                  // the reference stops earlier: the pass again, that far only
            __syncthreads();
            tile_pass(P, S, l, cur, src, ccur, q, restr, l2, false);
            if (!pass_sums(P, S, phase)) return false;
        }
        curs ^= 1u << l;
        done += q;
        src = SRC_U;
    }
    __syncthreads();
    if (threadIdx.x == 0) { S.pred[dir][l] = done; S.iter[l] += done; }
    __syncthreads();
    *res_out = res;
    return true;
}

// sor_big for a level in CTA 0's shared memory: the predicted number of sweeps (else two, then the
// rest) from a copy kept in the level's global buffer, the residuals of all of them summed
// together, and the sweeps taken again from the copy where the reference stops earlier.  Most
// stages take two sweeps or all ten, so a prediction rarely fails.
__device__ void sor_small(const MGP &P, MGShared &S, int l, int kmg, int dig, int dir, double *res_out) {
    const Patch &g = S.lev[l];
    const MGDev &L = P.L[l];
    // only as many warps as the level has nodes of one colour: idle warps cost issue slots and a
    // slower barrier
    const int T = min(MGT, (g.PS + 31) & ~31);
    if ((int)threadIdx.x < T) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = T >> 5;
        const int nn = 2 * g.PS, uo = g.uo;
        double *keep = L.u2;
        double res = 0.0, res_s = 0.0;
        const int nr = kmg == 1 && dig == 0 ? 1000000 : MG_NR;
        const int want = S.pred[dir][l];
        int done = 0;
        bool stop = false;
        while (!stop) {
            const int K = min(min(done < want ? want - done : (done ? 8 : 2), MG_NR), nr - done);
            const bool sure = done == 0 && dig != 0 && K <= 2;     // the second sweep is always taken
            if (!sure)
                for (int t = threadIdx.x; t < nn; t += T) keep[t] = smd[uo + t];
            team_sync(T);
            sweeps(P, g, L, K, T, false, false);
            team_sync(T);
            for (int k = warp; k < K; k += nw) {
                const double a = slot_sum(k, T);
                if (lane == 0) S.tot[k] = a;
            }
            team_sync(T);
            const int q = decide(P, S, K, done, nr, dig, res, res_s, stop);
            if (q < K) {
                for (int t = threadIdx.x; t < nn; t += T) smd[uo + t] = keep[t];
                team_sync(T);
                sweeps(P, g, L, q, T, false, false);
            }
            done += q;
            team_sync(T);
        }
        if (threadIdx.x == 0) { S.pred[dir][l] = done; S.iter[l] += done; S.res = res; }
    }
    __syncthreads();
    *res_out = S.res;
}

// a CTA-wide sum for CTA 0's own levels, outside the sweeps
__device__ double cta_sum(MGShared &S, double v) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    v = warp_sum(v);
    if (lane == 0) S.red[warp] = v;
    __syncthreads();
    double a = 0.0;
#pragma unroll
    for (int w = 0; w < MGW; w++) a = a + S.red[w];
    __syncthreads();
    return a;
}

// The part of a V-cycle on levels >= Ls, run by CTA 0: S(Ls)..R.. S*(ng-1) P.. S(Ls)
__device__ void small_region(const MGP &P, MGShared &S, int k, double *res) {
    const int ng = P.ng, Ls = P.Ls;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (Ls > 0) {     // the restricted residual of level Ls - 1 in, its correction from zeros
        const MGDev &L = P.L[Ls];
        const Patch g = level_patch(P, Ls);
        for (int j = warp; j < L.ny + 3; j += MGW)
            for (int i = lane; i < L.nx + 3; i += 32) {
                const int q = i + j * g.RP;
                g.u(q) = 0.0;
                if (i >= 1 && i <= L.nx + 1 && j >= 1 && j <= L.ny + 1) cp_async8(&g.b(q), L.b + (i - 1) + (j - 1) * (L.nx + 1));
            }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
    for (int l = Ls; l <= ng - 2; l++) {
        sor_small(P, S, l, k, l + 1 - ng, 0, res);
        // the residual into the slots' space (free between stages): the way up needs b again
        const Patch &g = S.lev[l], &c = S.lev[l + 1];
        residual_to(g, P.L[l], P.nmn, 0);
        for (int t = threadIdx.x; t < 2 * c.PS; t += MGT) smd[c.uo + t] = 0.0;
        __syncthreads();
        restriction(g, P.pbc, 0, [&](int i, int j) { return (int)c.m(i + j * c.RP); },
                    [&](int i, int j, double v) { c.b(i + j * c.RP) = v; });
        __syncthreads();
    }
    sor_small(P, S, ng - 1, k, 0, 0, res);
    for (int l = ng - 2; l >= Ls; l--) {
        const Patch &g = S.lev[l], &c = S.lev[l + 1];
        const int lg = lanes_of(g.RW), lpr = 1 << lg;
        const int ln = threadIdx.x & (lpr - 1), sub = threadIdx.x >> lg, nsub = MGT >> lg;
        for (int j = sub; j <= g.ny + 1; j += nsub)
            for (int i = ln; i <= g.nx + 1; i += lpr) {
                const int q = i + j * g.RP;
                if (g.m(q) <= 0) g.u(q) = prolonged(g.u(q), [&](int t) { return c.u(t); }, c.RP, i, j);
            }
        __syncthreads();
        sor_small(P, S, l, k, ng - l - 1, 1, res);
    }
    if (Ls > 0) {     // the correction out
        const MGDev &L = P.L[Ls];
        const Patch g = level_patch(P, Ls);
        for (int j = warp; j < L.ny + 3; j += MGW)
            for (int i = lane; i < L.nx + 3; i += 32) L.u[i + j * (L.nx + 3)] = g.u(i + j * g.RP);
    }
}

// iterative_solver.f90:18-66.  mode 0: stop on the reference's normalised L1 residual;
// mode 2: same cycles, stop on ||b-Au||_2/||b-Au_D||_2 <= eps.
__global__ void __launch_bounds__(MGT, 1) k_mg_solve(const __grid_constant__ MGP P) {
    __shared__ MGShared S;
    const int ng = P.ng, Ls = P.Ls;
    double res = 0.0, res_s = 0.0, rr = 0.0, bb = 0.0;
    unsigned curs = 0, phase = 0;       // each level's current buffer; sums taken so far
    for (int t = threadIdx.x; t < LEPIC_MAXLEV; t += MGT) { S.pred[0][t] = S.pred[1][t] = 0; S.iter[t] = 0; }
    const bool small = Ls < ng && blockIdx.x == 0;
    if (small) {                        // the coarse levels' masks (and level 0's u and b when it is one of them)
        for (int l = Ls; l < ng; l++) {
            const Patch g = level_patch(P, l);
            if (threadIdx.x == 0) S.lev[l] = g;
            const MGDev &L = P.L[l];
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            for (int j = warp; j < g.RH; j += MGW)
                for (int i = lane; i < g.RP; i += 32) {
                    const int q = i + j * g.RP;
                    const int n = i + j * g.RW;
                    g.m(q) = i < g.RW ? mask_of(g, L.bc[n], i, j, true) : M_WALL;
                    g.u(q) = l == 0 && i < g.RW ? L.u[n] : 0.0;
                    g.b(q) = l == 0 && i >= 1 && i <= L.nx + 1 && j >= 1 && j <= L.ny + 1 ? L.b[(i - 1) + (j - 1) * (L.nx + 1)] : 0.0;
                }
        }
    }
    __syncthreads();
    if (Ls == 0) {                      // one CTA holds the whole problem
        if (!grid_barrier(P.cnt, gridDim.x + P.bar_extra)) return;
        bb = cta_sum(S, wall_norm(level_patch(P, 0), P.L[0]));
    }
    int k = 1;
    bool conv = false, diverged = false;
    for (;;) {
        // mg.f90:85-225 -- one V-cycle; res is the L1 residual of the last finest-level sweep
        for (int l = 0; l < Ls && l <= ng - 2; l++) {
            const int src = l == 0 ? SRC_U : SRC_ZERO;
            if (!sor_big(P, S, l, k, l + 1 - ng, 0, src, true, false, k == 1 && l == 0, curs, &phase, &res, &bb)) return;
        }
        int top = Ls;
        if (Ls < ng) {
            curs &= ~(1u << Ls);        // the correction of level Ls is left in its first buffer
            if (small) {
                __syncthreads();
                small_region(P, S, k, &res);
            }
            if (Ls > 0 && !grid_barrier(P.cnt, gridDim.x + P.bar_extra)) return;
        } else {
            const int l = ng - 1;
            if (!sor_big(P, S, l, k, 0, 0, l == 0 ? SRC_U : SRC_ZERO, false, l == 0, k == 1 && l == 0, curs, &phase,
                         &res, &bb)) return;
            top = ng - 1;
        }
        for (int l = top - 1; l >= 0; l--)
            if (!sor_big(P, S, l, k, ng - l - 1, 1, SRC_UP, false, l == 0, false, curs, &phase, &res, &bb)) return;
        if (Ls == 0) {
            double a = 0.0, q2 = 0.0;
            last_residual(level_patch(P, 0), P.L[0], a, q2, MGT, false, true);
            rr = cta_sum(S, q2);
        } else {
            rr = S.tot[MG_KMAX];
        }
        res = res / P.alpha;
        if (k == 1) res_s = res;
        else if (fabs(res / res_s) > 10.0) { diverged = true; break; }
        if (P.mode == 2) conv = sqrt(rr) <= P.eps * sqrt(bb);
        else conv = res <= P.eps;
        if (conv || k == P.ncycl) break;
        k = k + 1;
    }
    // the potential into phi
    if (Ls == 0) {
        const Patch g = level_patch(P, 0);
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int j = warp; j < g.RH; j += MGW)
            for (int i = lane; i < g.RW; i += 32) P.L[0].u[i + j * g.RW] = g.u(i + j * g.RP);
    } else if (curs & 1u) {
        const long long nn = (long long)(P.L[0].nx + 3) * (P.L[0].ny + 3);
        for (long long t = blockIdx.x * (long long)MGT + threadIdx.x; t < nn; t += (long long)gridDim.x * MGT)
            P.L[0].u[t] = P.L[0].u2[t];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (diverged) { set_err(P.cnt, LERR_DIVERGED, 500); return; }
        // ncycl cycles without reaching eps: the reference goes on with this potential
        // (iterative_solver.f90:56); the call reports it and phi holds the last cycle's result
        if (!conv) set_err(P.cnt, LERR_NOTCONV, 501);
        double ktot = 0.0;
        for (int i = 1; i <= ng; i++) ktot = ktot + (double)S.iter[i - 1] / pow(2.0, 2 * (i - 1));
        P.cnt->mg_cycles = k;
        P.cnt->mg_sweeps_fine = S.iter[0];
        P.cnt->mg_res_l1 = res;
        P.cnt->mg_ktot = ktot;
        P.cnt->mg_res_l2 = sqrt(rr);
        P.cnt->mg_b_l2 = sqrt(bb);
    }
}

// ---------------------------------------------------------------------------------------
// The levels of at most lepic_options::mg_small_nodes nodes are CTA 0's, as far as its shared memory
// holds them (one level of up to about 4900 nodes and the coarser ones).  The default of 2000 is
// where one CTA's sweep, bound by its SM's shared-memory loads and FP64 units, costs as much as a
// tile pass over the whole GPU with its grid barrier: 65^2 nodes take 11.4 / 35 us for a stage of
// 2 / 10 sweeps on CTA 0 and 10 / 33 us in tiles (128^2 solve 0.69 against 0.64 ms), 49 x 33 nodes
// are 5 % of the 384 x 256 solve faster on CTA 0, 33^2 nodes 10 % of the 128^2 solve.
#define MG_SMEM (224 * 1024)   // dynamic shared memory per CTA (one per SM)

// The kernel's parameters but for a solve's own (mg_solve): the split of the levels and their tiles,
// which follow from the deck and the options and take about 6 us per tiled level to choose.
static MGP mg_params(const lepic_ctx *c) {
    MGP P;
    memset(&P, 0, sizeof(P));
    const double eps0 = c->cfg.eps0;
    for (int l = 0; l < c->nlev; l++) {
        const MGLevel &a = c->lev[l];
        MGDev &d = P.L[l];
        d.nx = a.nx; d.ny = a.ny;
        d.aw = eps0 / (a.hx * a.hx);
        d.an = eps0 / (a.hy * a.hy);
        d.ac = -(d.an + d.an + d.aw + d.aw);
        d.y = fabs(d.ac) > 1e-30 && fabs(d.ac) < 1e30 ? 1.0 / d.ac : 0.0;
        d.u = a.u; d.b = a.b; d.bc = a.bc;
        // With an odd number of rows between periodic edges (only the coarsest level of a deck can
        // have one) the nodes across the edge have the colour of their neighbours, and nodes of row
        // ny + 1 whose residual counts are overwritten by the copy after their update: in both cases
        // a half-sweep's residuals are not final before the edge rows are copied
        d.seam = c->cfg.flag_pbc && ((a.ny & 1) || a.top_counts);
        d.u2 = l == 0 ? c->cg_ap : a.u2;
    }
    P.ng = c->nlev;
    // the CTA-0 part: the coarsest levels, as long as each has at most mg_small_nodes nodes and they
    // fit in shared memory together (a level's residual in the slots' space)
    const long long small_nodes = c->opt.mg_small_nodes;
    const long long room = MG_SMEM / 8 - MG_SLOTS;      // doubles
    long long total = 0;                                // nodes of the CTA-0 part, both colours' padding included
    P.Ls = c->nlev;
    auto padded = [&](int l) { return mg_level_len(c->lev[l].nx, c->lev[l].ny); };
    for (int l = c->nlev - 1; l >= 0; l--) {
        const MGLevel &a = c->lev[l];
        if ((long long)(a.nx + 1) * (a.ny + 1) > small_nodes || padded(l) > MG_SLOTS ||
            17 * (total + padded(l)) + 16 > 8 * room) break;
        total += padded(l);
        P.Ls = l;
    }
    long long off = 0;
    for (int l = P.Ls; l < c->nlev; l++) {
        P.L[l].su = (int)off;
        P.L[l].sb = (int)(off + total);
        P.L[l].sm = (int)(16 * total + off);
        off += padded(l);
    }
    // per level the tile that ends a pass soonest: its tiles go round the grid's CTAs, so a pass
    // lasts (rounds) x (a tile's sweeps over its region, halo included, plus its fixed latencies,
    // which cost about as much as 1500 nodes)
    P.cap = (int)(8 * room / 17 / 16 * 16);
    const int workers = std::max(1, c->mg_grid - (P.Ls < c->nlev ? 1 : 0));
    for (int l = 0; l < P.Ls; l++) {
        double best = -1.0;
        for (int tx = 8; tx <= 128; tx += 4)
            for (int ty = 4; ty <= 128; ty += 4) {
                const long long region = (long long)((tx + 2 * MG_HMAX) | 1) * (ty + 2 * MG_HMAX + 4) + 2;
                if (region > P.cap) continue;
                const long long nt = (long long)((c->lev[l].nx + tx) / tx) * ((c->lev[l].ny + ty) / ty);
                const double rounds = (double)((nt + workers - 1) / workers);
                const double cost = rounds * ((double)region + 1500.0);
                if (best < 0.0 || cost < best) { best = cost; P.L[l].tx = tx; P.L[l].ty = ty; }
            }
    }
    P.omega = c->cfg.omega;
    P.alpha = fabs((double)(c->cfg.nx + 1) * (c->cfg.ny + 1) * P.L[0].ac) * 1.0;
    P.ncycl = c->cfg.ncycl;
    P.pbc = c->cfg.flag_pbc;
    P.nmn = c->cfg.flag_nmn;
    P.partials = c->partials;
    P.cnt = c->dcnt;
    return P;
}

// the plan of a context's solves: at its creation, and again when an option it depends on changes
int mg_init(lepic_ctx *c) {
    int occ = 0;
    LCUDA(cudaFuncSetAttribute(k_mg_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, MG_SMEM));
    LCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_mg_solve, MGT, MG_SMEM));
    if (occ < 1) { c->last_err = "multigrid kernel does not fit on an SM"; return LEPIC_ECUDA; }
    c->mg_grid = c->num_sms;       // a CTA takes an SM's shared memory
    const MGP P = mg_params(c);
    for (int l = P.Ls; l < P.ng; l++)
        if (c->lev[l].u2_len < mg_level_len(P.L[l].nx, P.L[l].ny)) {   // a stage keeps its start there
            c->last_err = "multigrid: a level's second buffer is too short";
            return LEPIC_ECUDA;
        }
    if (!c->mg_plan && !(c->mg_plan = malloc(sizeof(MGP)))) { c->last_err = "multigrid: no memory for its plan"; return LEPIC_ENOMEM; }
    memcpy(c->mg_plan, &P, sizeof(P));
    return LEPIC_OK;
}

int mg_solve(lepic_ctx *c, double eps, int mode) {
    MGP P;
    memcpy(&P, c->mg_plan, sizeof(P));
    P.eps = eps;
    P.mode = mode;
    P.bar_extra = (unsigned)c->opt.barrier_extra;
    void *args[] = {&P};
    LCUDA(cudaMemsetAsync(&c->dcnt->bar_arrived, 0, sizeof(unsigned long long) + sizeof(int), c->stream));
    LCUDA(cudaLaunchCooperativeKernel((void *)k_mg_solve, dim3(P.Ls == 0 ? 1 : c->mg_grid), dim3(MGT), args, MG_SMEM, c->stream));
    return LEPIC_OK;
}
