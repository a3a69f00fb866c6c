// The coarse part of a multigrid V-cycle (or, on small grids, all of it) in
// one thread-block cluster with every level's arrays in shared memory.
//
// A level is cut into slabs of q planes in z, one slab per CTA.  Each CTA
// holds its slab of x with one ghost layer on every side, of r, and with
// variable density of 1/rho; the residual of the level being restricted has
// one buffer for all levels.  A colour pass reads shared memory only, writes
// the new values home and, for the first and last plane of the slab, into
// the neighbours' ghost planes (distributed shared memory).  It ends when the
// neighbours' values of the pass have arrived, counted on an mbarrier, or, with
// periodic images within the planes, at the hardware cluster barrier.  Ghost
// columns and rows hold the periodic images, or zero beyond a wall; adding a
// zero term leaves every sum's bits alone, so boundary and interior points run
// the same loads and the boundary rules reduce to coefficients.  Every point's
// sum has the order of the per-phase kernels (mg_ops.cuh): the same bits as one
// launch per phase.
//
// What bounds it: these levels have 10^2..10^5 points, and a phase issued as
// its own launch costs the launch and one or two dependent L2 latencies
// (2.5-4 us) whatever its size.  Here a phase costs its points' instructions
// on 16 SMs and a hand-over: 0.45-1.2 us a colour pass, of which 0.15-0.3 us
// is the wait for the neighbours (a full cluster barrier measured 0.3 us).
// Measured on a B200: the V(2,1) part from 33^3 down, FP32, 47 us against
// about 120 us for its 34 launches, MAC from 32^3 27 against 65 us; a
// 16^3 FP64 cavity step 761 -> 430 us, a 64^3 mixed step with a sphere
// 1.41 -> 1.21 ms.
//
// Along x the points are stored split by parity (even columns first), so that
// a colour pass and its x neighbours read consecutive words; stride-2 reads
// would hit every second bank.
//
// Within a colour pass no CTA reads a value another one writes: the colours
// are exact Gauss-Seidel colours (coupled points never share one).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#ifndef RMT3D_HOST_SIM  // the host-thread check brings its own primitives
#include "cluster_ops.cuh"
#endif
#include "mg.h"
#include "mg_ops.cuh"

namespace rmt3d {

// Threads per CTA.  512 measured fastest, in an earlier form whose warps all
// polled for the neighbours: the V(2,1) part of a 33^3 FP32 hierarchy took 49 us,
// against 56 us with 256 and 53 us with 1024 threads (whose 64 registers spill).
#ifndef RMT3D_SLAB_THREADS
#define RMT3D_SLAB_THREADS 512
#endif
constexpr int kSlabThreads = RMT3D_SLAB_THREADS;

// t / d by the precomputed inv = ceil(2^31 / d): (t + 1/2) / d is at least
// 1 / (2 d) away from an integer, so the quotient is exact while
// (2 t + 1) d < 2^31
__device__ __forceinline__ int fdiv(int t, unsigned inv) { return (int)__umulhi((unsigned)(2 * t + 1), inv); }

template <typename T>
struct slab_ctx {
    T *sm;             // this CTA's shared memory
    int rank, tid;
    uint64_t *bar;     // two mbarriers for the neighbours' values, used in turn
    int *failed;       // a wait on one of them gave up (set by the thread that waits)
};

// offset of column i within a row: columns -1..n0 as i+1, even ones first
__device__ __forceinline__ int col(const slab_level &L, int i) {
    const int q = i + 1;
    return (q & 1) * L.H + (q >> 1);
}
__device__ __forceinline__ int nplanes(const slab_level &L, int rank) {
    const int left = L.n2 - rank * L.q;
    return left < 0 ? 0 : (left < L.q ? left : L.q);
}

// A level as a CTA works on it, in registers.  (The layout lies in the
// kernel's constant parameters; `keep` stops the compiler from fetching a
// value again at every use, which had cost a third of the instructions.)
__device__ __forceinline__ int keep(int v) {
    asm("" : "+r"(v));
    return v;
}
template <typename T>
struct slab_view {
    int np, k0;          // planes here, the first one's index
    int klo, khi;        // the level's first / last plane in z, or -1
    int n0, n1, RS, PX, PR, H;
    int ox, orr, os, oi; // of plane 0 (x and 1/rho: past the lower ghost plane)
    bool p0, p1, p2;
    // the ghost planes of the slabs below and above that mirror this slab's
    // first and last plane (kdn, kup; -1: a wall): generic pointers, and for
    // sends the shared::cluster addresses with the receivers' mbarriers
    int kdn, kup;
    T *dn, *up;
    cl_addr sdn, sup, bdn, bup;
    bool async;  // rim values go as sends (no periodic images within a plane)
};
template <typename T>
__device__ __forceinline__ slab_view<T> view_of(const slab_ctx<T> &C, const slab_level &L) {
    slab_view<T> V;
    V.np = keep(nplanes(L, C.rank));
    V.k0 = keep(C.rank * L.q);
    const int k1 = V.k0 + V.np;
    V.klo = keep(V.k0 == 0 ? 0 : -1);
    V.khi = keep(k1 == L.n2 ? V.np - 1 : -1);
    V.n0 = keep(L.n0), V.n1 = keep(L.n1);
    V.RS = keep(L.RS), V.PX = keep(L.PX), V.PR = keep(L.PR), V.H = keep(L.H);
    V.ox = keep(L.ox + L.PX), V.orr = keep(L.orr), V.os = keep(L.os), V.oi = keep(L.oi + L.PX);
    V.p0 = L.p0, V.p1 = L.p1, V.p2 = L.p2;
    V.kdn = V.kup = -1;
    V.dn = V.up = nullptr;
    V.sdn = V.sup = V.bdn = V.bup = 0;
    V.async = !(L.p0 || L.p1);
    if (V.np > 0) {
        if (V.k0 > 0 || L.p2) {
            const int rk = V.k0 > 0 ? C.rank - 1 : (L.n2 - 1) / L.q, o = L.ox + (nplanes(L, rk) + 1) * L.PX;
            V.kdn = 0;
            V.dn = cl_map(C.sm, rk) + o;
            V.sdn = cl_remote(C.sm + o, rk);
            V.bdn = cl_remote(C.bar, rk);
        }
        if (k1 < L.n2 || L.p2) {
            const int rk = k1 < L.n2 ? C.rank + 1 : 0;
            V.kup = V.np - 1;
            V.up = cl_map(C.sm, rk) + L.ox;
            V.sup = cl_remote(C.sm + L.ox, rk);
            V.bup = cl_remote(C.bar, rk);
        }
    }
    V.kdn = keep(V.kdn);
    V.kup = keep(V.kup);
    return V;
}

// v at element o = (i, j) of a plane of x and, on periodic axes, its images
template <typename T>
__device__ __forceinline__ void put_images(const slab_view<T> &V, T *plane, int i, int j, int o, T v) {
    const bool gi = V.p0 && (i == 0 || i == V.n0 - 1), gj = V.p1 && (j == 0 || j == V.n1 - 1);
    // column n0 mirrors 0 and column -1 mirrors n0-1; rows alike
    auto cc = [&](int q) { return (q & 1) * V.H + (q >> 1); };
    const int di = (i == 0 ? cc(V.n0 + 1) : cc(0)) - cc(i + 1);
    const int dj = (j == 0 ? V.n1 : -V.n1) * V.RS;
    plane[o] = v;
    if (gi) plane[o + di] = v;
    if (gj) plane[o + dj] = v;
    if (gi && gj) plane[o + di + dj] = v;
}

// x = v at element o = (i, j) of plane kl: home, the periodic images (EDGE:
// the point may lie on the rim of its plane) and the neighbours' ghost
// planes, there as sends on mbarrier `use` & 1 (use >= 0) or plain stores
template <typename T, bool EDGE>
__device__ __forceinline__ void put_x(const slab_ctx<T> &C, const slab_view<T> &V, int i, int j, int kl, int o, T v,
                                      int use) {
    T *home = C.sm + (V.ox + kl * V.PX);
    if (EDGE && (V.p0 | V.p1)) {
        put_images(V, home, i, j, o, v);
        if (kl == V.kdn) put_images(V, V.dn, i, j, o, v);
        if (kl == V.kup) put_images(V, V.up, i, j, o, v);
    } else {
        home[o] = v;
        if (use >= 0) {
            const unsigned at = (unsigned)o * sizeof(T), bo = (use & 1) * sizeof(uint64_t);
            if (kl == V.kdn) cl_send(V.sdn + at, v, V.bdn + bo);
            if (kl == V.kup) cl_send(V.sup + at, v, V.bup + bo);
        } else {
            if (kl == V.kdn) V.dn[o] = v;
            if (kl == V.kup) V.up[o] = v;
        }
    }
}

// ---- FEM: one node ---------------------------------------------------------
// MODE 0: Gauss-Seidel update of x; MODE 1: residual into the residual buffer.
// EDGE: the node may lie on the rim of its plane (its sum then runs term by
// term, as the general path of fem_offdiag does); the interior of a plane and
// its rim are separate work items, so a warp follows one of the two.
// o: the node's element within a plane of x; dm: from its column to column
// i-1 (column i+1 follows it).
template <typename T, bool VD, int MODE, bool EDGE>
__device__ __forceinline__ void fem_node(const slab_ctx<T> &C, const slab_view<T> &V, int i, int j, int kl, int o,
                                         int dm, int use) {
    const T *x0 = C.sm + (V.ox + kl * V.PX + o), *xm = x0 - V.PX, *xp = x0 + V.PX;
    const T *xmm = xm - V.RS, *xmp = xm + V.RS, *xpm = xp - V.RS, *xpp = xp + V.RS;
    const int ro = kl * V.PR + o - V.RS;
    const T rv = C.sm[V.orr + ro];
    const T a10 = xmm[0], a12 = xmp[0], d10 = xpm[0], d12 = xpp[0];
    xmm += dm, xmp += dm, xpm += dm, xpp += dm;
    const T *ym = x0 - V.RS + dm, *yp = x0 + V.RS + dm;
    const T a00 = xmm[0], a20 = xmm[1], a02 = xmp[0], a22 = xmp[1];
    const T d00 = xpm[0], d20 = xpm[1], d02 = xpp[0], d22 = xpp[1];
    const T a01 = xm[dm], a21 = xm[dm + 1], d01 = xp[dm], d21 = xp[dm + 1];
    const T b00 = ym[0], b20 = ym[1], b02 = yp[0], b22 = yp[1];
    const bool b2 = kl == V.klo || kl == V.khi;
    T s, diag;
    if (VD) {
        // 1/rho of the eight cells around the node: lower and upper layer,
        // (y, x); zero outside the box.  Cell columns i-1, i; rows j-1, j.
        const T *r2 = C.sm + (V.oi + kl * V.PX + o), *r1 = r2 - V.PX;
        const T u10 = r1[-V.RS], u11 = r1[0], u00 = r1[dm - V.RS], u01 = r1[dm];
        const T v10 = r2[-V.RS], v11 = r2[0], v00 = r2[dm - V.RS], v01 = r2[dm];
        // corners -1/rho, edges -(sum of the two cells), in (z, y, x) order:
        // -2 times the mean of two cells, and -1 times the one cell where a
        // wall leaves only one, are that sum exactly
        s = 0;
        s += -u00 * a00;
        s += -(u00 + u10) * a10;
        s += -u10 * a20;
        s += -(u00 + u01) * a01;
        s += -(u10 + u11) * a21;
        s += -u01 * a02;
        s += -(u01 + u11) * a12;
        s += -u11 * a22;
        s += -(u00 + v00) * b00;
        s += -(u10 + v10) * b20;
        s += -(u01 + v01) * b02;
        s += -(u11 + v11) * b22;
        s += -v00 * d00;
        s += -(v00 + v10) * d10;
        s += -v10 * d20;
        s += -(v00 + v01) * d01;
        s += -(v10 + v11) * d21;
        s += -v01 * d02;
        s += -(v01 + v11) * d12;
        s += -v11 * d22;
        T c8 = 0;
        c8 += u00;
        c8 += u10;
        c8 += u01;
        c8 += u11;
        c8 += v00;
        c8 += v10;
        c8 += v01;
        c8 += v11;
        diag = (T)4 * c8;  // 32 x their mean, halved per wall: exactly this
    } else if (!EDGE && !b2) {
        T e = (b00 + b20) + (b02 + b22);
        e += (a01 + a21) + (a10 + a12);
        e += (d01 + d21) + (d10 + d12);
        T q = (a00 + a20) + (a02 + a22);
        q += (d00 + d20) + (d02 + d22);
        s = (T)-2 * e - q;
        diag = MODE == 1 ? (T)32 : (T)0.03125;
    } else {
        // planes next to a periodic seam sum term by term too
        const bool b0 = EDGE && !V.p0 && (i == 0 || i == V.n0 - 1), b1 = EDGE && !V.p1 && (j == 0 || j == V.n1 - 1);
        const bool w2 = b2 && !V.p2;
        const T ex = b0 ? (T)-1 : (T)-2, ey = b1 ? (T)-1 : (T)-2, ez = w2 ? (T)-1 : (T)-2;
        s = 0;
        s += -a00;
        s += ex * a10;
        s += -a20;
        s += ey * a01;
        s += ey * a21;
        s += -a02;
        s += ex * a12;
        s += -a22;
        s += ez * b00;
        s += ez * b20;
        s += ez * b02;
        s += ez * b22;
        s += -d00;
        s += ex * d10;
        s += -d20;
        s += ey * d01;
        s += ey * d21;
        s += -d02;
        s += ex * d12;
        s += -d22;
        const int h = (b0 ? 1 : 0) + (b1 ? 1 : 0) + (w2 ? 1 : 0);
        diag = MODE == 1 ? (T)(32 >> h) : (T)(1 << h) * (T)0.03125;
    }
    if (MODE == 1) C.sm[V.os + ro] = rv - s - diag * x0[0];
    else put_x<T, EDGE>(C, V, i, j, kl, o, VD ? (rv - s) / diag : (rv - s) * diag, use);
}

// ---- MAC: one cell ---------------------------------------------------------
template <typename T, bool VD, int MODE>
__device__ __forceinline__ void mac_cell(const slab_ctx<T> &C, const slab_view<T> &V, int i, int j, int kl, int o,
                                         int dm, int use) {
    const T *x = C.sm + (V.ox + kl * V.PX + o);
    const T xm = x[dm], xp = x[dm + 1], ym = x[-V.RS], yp = x[V.RS], zm = x[-V.PX], zp = x[V.PX];
    const int ro = kl * V.PR + o - V.RS;
    const T rv = C.sm[V.orr + ro];
    const bool i0 = i == 0, i1 = i == V.n0 - 1, j0 = j == 0, j1 = j == V.n1 - 1, z0 = kl == V.klo, z1 = kl == V.khi;
    const bool mx = !i0 || V.p0, px = !i1 || V.p0, my = !j0 || V.p1, py = !j1 || V.p1, mz = !z0 || V.p2,
               pz = !z1 || V.p2;
    T s, diag;
    if (VD) {
        const T *ri = C.sm + (V.oi + kl * V.PX + o);
        const T rc = ri[0];
        const T ax1 = mx ? (T)0.5 * (ri[dm] + rc) : (T)0, ax2 = px ? (T)0.5 * (rc + ri[dm + 1]) : (T)0;
        const T ay1 = my ? (T)0.5 * (ri[-V.RS] + rc) : (T)0, ay2 = py ? (T)0.5 * (rc + ri[V.RS]) : (T)0;
        const T az1 = mz ? (T)0.5 * (ri[-V.PX] + rc) : (T)0, az2 = pz ? (T)0.5 * (rc + ri[V.PX]) : (T)0;
        T csum = 0;
        s = 0;
        s += ax1 * xm + ax2 * xp;
        csum += ax1 + ax2;
        s += ay1 * ym + ay2 * yp;
        csum += ay1 + ay2;
        s += az1 * zm + az2 * zp;
        csum += az1 + az2;
        const int cnt = (mx ? 1 : 0) + (px ? 1 : 0) + (my ? 1 : 0) + (py ? 1 : 0) + (mz ? 1 : 0) + (pz ? 1 : 0);
        diag = (T)(-cnt) * (csum / (T)cnt);
    } else {
        // both orders of summation: cheaper than a warp running both paths
        const bool in = !(i0 | i1 | j0 | j1 | z0 | z1);
        const T s1 = ((xm + xp) + (ym + yp)) + (zm + zp);
        const T s2 = ((((xm + xp) + ym) + yp) + zm) + zp;
        s = in ? s1 : s2;
        const int missing = (mx ? 0 : 1) + (px ? 0 : 1) + (my ? 0 : 1) + (py ? 0 : 1) + (mz ? 0 : 1) + (pz ? 0 : 1);
        diag = (T)(-6 + missing);
    }
    if (MODE == 1) C.sm[V.os + ro] = rv - s - diag * x[0];
    else put_x<T, true>(C, V, i, j, kl, o, (rv - s) / diag, use);
}

// What a colour pass of a level needs to deal out its points, worked out once
// per launch and kept in shared memory: a pass is short, and every warp would
// otherwise spend more on this than on its points.
struct alignas(16) slab_pass {
    // FEM: work items are the colour's interior nodes of every plane, rounded
    // up to whole warps (tin), then its rim nodes; MAC: nin cells a row
    int tin, tot, nin;
    unsigned inv_nin;
    int xin;
    unsigned inv_xin;
    int base, dm;  // first interior node's element; from a node's column to column i-1
    int R2, bytes;  // two rows; bytes of rim values to expect from the neighbours
    int xn, yn;
    int nrim;
    unsigned inv_rim;
    int lo, c00;   // whether the first column (bit 0), row (bit 1) is on the rim; element of node (0, 0)
    int rim_rows;  // rim nodes in whole rows
    int pad[3];
};

// points of a colour in plane k
template <int KIND>
__device__ __forceinline__ int colour_points(const slab_level &L, int colour, int k) {
    if (KIND == 1) return L.cx[colour & 1].n * L.cy[colour >> 1].n;
    return (L.n0 * L.n1 + (((k + colour) & 1) ? 0 : 1)) >> 1;
}

template <typename T, int KIND>
__device__ __forceinline__ void make_pass(const slab_level &L, int rank, int colour, slab_pass *out) {
    slab_pass P;
    const int np = nplanes(L, rank), k0 = rank * L.q;
    if (KIND == 1) {
        const int ci = colour & 1, cj = colour >> 1;
        const slab_col &X = L.cx[ci], &Y = L.cy[cj];
        P.nin = X.in * Y.in;
        P.nrim = X.n * Y.n - P.nin;
        P.tin = (P.nin * np + 31) & ~31;
        P.tot = P.tin + P.nrim * np;
        P.inv_nin = L.inv_in[colour];
        P.inv_rim = L.inv_rim[colour];
        P.xin = X.in;
        P.inv_xin = X.inv_in;
        P.xn = X.n;
        P.yn = Y.n;
        P.lo = X.lo | (Y.lo << 1);
        P.rim_rows = (Y.n - Y.in) * X.n;
        P.R2 = 2 * L.RS;
        // column i of parity ci is element i / 2 + (ci ? 1 : H) of its row
        P.c00 = (ci ? 1 : L.H) + (cj + 1) * L.RS;
        P.base = P.c00 + Y.lo * P.R2 + X.lo;
        P.dm = ci ? L.H - 1 : -L.H;
    } else {
        P.nin = (L.n0 + 1) >> 1;
        P.inv_nin = L.inv_half;
        P.xin = L.n1;
        P.inv_xin = L.inv_n1;
        P.tin = P.tot = P.nin * L.n1 * np;
        P.base = P.dm = P.R2 = P.xn = P.yn = P.lo = P.c00 = P.nrim = P.rim_rows = 0;
        P.inv_rim = 0;
    }
    int n = 0;
    if (np > 0) {
        if (k0 > 0 || L.p2) n += colour_points<KIND>(L, colour, k0 > 0 ? k0 - 1 : L.n2 - 1);
        if (k0 + np < L.n2 || L.p2) n += colour_points<KIND>(L, colour, k0 + np < L.n2 ? k0 + np : 0);
    }
    P.bytes = n * (int)sizeof(T);
    *out = P;
}

// one colour pass (MODE 0) or the residual of one colour's points (MODE 1)
template <typename T, int KIND, bool VD, int MODE>
__device__ __forceinline__ void colour_pass(const slab_ctx<T> &C, const slab_pass &table, const slab_view<T> &V,
                                            int colour, int use) {
    if (C.tid >= table.tot) return;
    const slab_pass P = table;  // in registers: the stores below could alias it
    if (KIND == 1) {
        for (int t = C.tid; t < P.tot; t += kSlabThreads) {
            if (t < P.tin) {
                const int kl = fdiv(t, P.inv_nin);
                if (kl >= V.np) continue;
                const int u = t - kl * P.nin, b = fdiv(u, P.inv_xin);
                fem_node<T, VD, MODE, false>(C, V, 0, 0, kl, P.base + b * P.R2 + (u - b * P.xin), P.dm, use);
            } else {
                const int e = t - P.tin, kl = fdiv(e, P.inv_rim);
                const int ylo = P.lo >> 1, xlo = P.lo & 1;
                int u = e - kl * P.nrim, a, b;
                const int rows = P.rim_rows;  // whole rim rows first
                if (u < rows) {
                    const int rr = u >= P.xn;
                    a = u - (rr ? P.xn : 0);
                    b = rr < ylo ? 0 : P.yn - 1;
                } else {
                    u -= rows;
                    const int two = P.xn - P.xin == 2;  // 1 or 2 rim nodes of each other row
                    b = ylo + (two ? u >> 1 : u);
                    a = (two ? u & 1 : 0) < xlo ? 0 : P.xn - 1;
                }
                fem_node<T, VD, MODE, true>(C, V, 2 * a + (colour & 1), 2 * b + (colour >> 1), kl,
                                            P.c00 + b * P.R2 + a, P.dm, use);
            }
        }
    } else {
        for (int t = C.tid; t < P.tot; t += kSlabThreads) {
            const int row = fdiv(t, P.inv_nin), a = t - row * P.nin;
            const int kl = fdiv(row, P.inv_xin), j = row - kl * P.xin;
            const int ci = (j + V.k0 + kl + colour) & 1, i = 2 * a + ci;
            if (i < V.n0)
                mac_cell<T, VD, MODE>(C, V, i, j, kl, (j + 1) * V.RS + a + (ci ? 1 : V.H), ci ? V.H - 1 : -V.H, use);
        }
    }
}

// Sweeps of a level.  A pass ends when this CTA is done and its neighbours'
// rim values of the pass have arrived (or, with periodic images within the
// planes, at the cluster barrier).  A neighbour may run one pass ahead -- it
// then has all this CTA's rim values, so the ghost plane it writes has been
// read -- hence two mbarriers in turn.  `use` counts the passes of the whole
// cluster; CTAs without planes take part with nothing to wait for.  After a wait
// that gave up a CTA sends its values on, so that no other waits for it, but
// neither waits nor arms: the phase it gave up on may still be open, and a
// second arrival in it is not allowed.
template <typename T, int KIND, bool VD>
__device__ __forceinline__ void smooth_level(const slab_ctx<T> &C, const slab_view<T> &V,
                                             int sweeps, const slab_pass *P, int &use) {
    constexpr int nc = KIND == 1 ? 4 : 2;
    for (int s = 0; s < sweeps * nc; s++) {
        const int colour = s % nc;
        if (V.async) {
            uint64_t *bar = C.bar + (use & 1);
            // one thread of the last warp, which has the fewest points, waits for
            // the neighbours; the block barrier hands on what it saw (every
            // warp polling cost a quarter of a pass's issue slots).  It arms here
            // too: values that came before lower the phase's byte count below zero
            // and cannot end it, as its one arrival is still due.
            colour_pass<T, KIND, VD, 0>(C, P[colour], V, colour, use);
            if (C.tid == kSlabThreads - 1 && *C.failed == 0) {
                halo_arm(bar, P[colour].bytes);
                if (!halo_wait(bar, (use >> 1) & 1)) *C.failed = 1;
            }
            __syncthreads();
            use++;
        } else {
            colour_pass<T, KIND, VD, 0>(C, P[colour], V, colour, -1);
            cl_barrier();
        }
    }
}

__device__ __forceinline__ int min2(int a, int b) { return a < b ? a : b; }

// plane k of the fine residual, wherever in the cluster it is
template <typename T>
__device__ __forceinline__ const T *res_plane(const slab_ctx<T> &C, const slab_level &F, int k) {
    const int rk = fdiv(k, F.inv_q);
    return cl_map(C.sm, rk) + F.os + (k - rk * F.q) * F.PR;
}

// The coarse right-hand side from the fine residual.  A CTA computes the
// coarse planes whose fine plane 2 K it holds (most of what they read) and
// writes them where they live; the coarsest level's go to every CTA, in FP64,
// as the dense solve reads them.
template <typename T, int KIND>
__device__ __forceinline__ void restrict_level(const slab_ctx<T> &C, const slab_args &S, const slab_level &F,
                                               const slab_level &K, bool last) {
    const int f0 = C.rank * F.q, f1 = f0 + nplanes(F, C.rank);
    const int K0 = (f0 + 1) >> 1, K1 = min2((f1 + 1) >> 1, K.n2);
    const int tot = K.n0 * K.n1 * (K1 - K0);
    for (int t = C.tid; t < tot; t += kSlabThreads) {
        const int row = fdiv(t, K.inv_n0), I = t - row * K.n0;
        const int kc = fdiv(row, K.inv_n1), J = row - kc * K.n1, kk = K0 + kc;
        T s = 0;
        if (KIND == 0) {
            const int c0 = col(F, 2 * I), c1 = col(F, 2 * I + 1);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const T *r = res_plane(C, F, 2 * kk + c) + 2 * J * F.RS;
                s += r[c0];
                s += r[c1];
                s += r[c0 + F.RS];
                s += r[c1 + F.RS];
            }
        } else {
            // a neighbour beyond a wall has weight zero (any stored value in
            // its place)
            int cx[3], cy[3], cz[3];
            T wx[3], wy[3], wz[3];
#pragma unroll
            for (int o = 0; o < 3; o++) {
                const T w = o == 1 ? (T)1 : (T)0.5;
                const int xx = wrapi(2 * I + o - 1, F.n0, F.p0), yy = wrapi(2 * J + o - 1, F.n1, F.p1),
                          zz = wrapi(2 * kk + o - 1, F.n2, F.p2);
                cx[o] = col(F, xx < 0 ? 2 * I : xx);
                cy[o] = (yy < 0 ? 2 * J : yy) * F.RS;
                cz[o] = zz < 0 ? 2 * kk : zz;
                wx[o] = xx < 0 ? (T)0 : w;
                wy[o] = yy < 0 ? (T)0 : w;
                wz[o] = zz < 0 ? (T)0 : w;
            }
#pragma unroll
            for (int oc = 0; oc < 3; oc++) {
                const T *pl = res_plane(C, F, cz[oc]);
#pragma unroll
                for (int ob = 0; ob < 3; ob++) {
                    const T *r = pl + cy[ob];
#pragma unroll
                    for (int oa = 0; oa < 3; oa++) s += wx[oa] * wy[ob] * wz[oc] * r[cx[oa]];
                }
            }
        }
        const T v = (T)0.5 * s;
        if (last) {
            double *rs = reinterpret_cast<double *>(reinterpret_cast<unsigned char *>(C.sm) + S.dense_off);
            for (int rk = 0; rk < S.csize; rk++) cl_map(rs, rk)[I + K.n0 * (J + K.n1 * kk)] = (double)v;
        } else {
            const int rk = fdiv(kk, K.inv_q);
            cl_map(C.sm, rk)[K.orr + (kk - rk * K.q) * K.PR + J * K.RS + col(K, I)] = v;
        }
    }
}

// x of the fine level += the interpolated coarse x, four fine points of a
// plane per work item (they share their coarse values)
template <typename T, int KIND>
__device__ __forceinline__ void prolong_level(const slab_ctx<T> &C, const slab_level &F, const slab_level &K,
                                              const slab_view<T> &V) {
    const int tot = K.n0 * K.n1 * V.np, k0 = V.k0;
    for (int t = C.tid; t < tot; t += kSlabThreads) {
        const int row = fdiv(t, K.inv_n0), I = t - row * K.n0;
        const int kl = fdiv(row, K.inv_n1), J = row - kl * K.n1;
        const int k = k0 + kl, k2 = k >> 1;
        // coarse planes and their weights
        int kz[2] = {k2, k2};
        T wz[2] = {1, 0};
        if (KIND == 0) {
            const int o = wrapi(k2 + ((k & 1) ? 1 : -1), K.n2, K.p2);
            if (o >= 0) {
                kz[1] = o;
                wz[0] = (T)0.75;
                wz[1] = (T)0.25;
            }
        } else if (k & 1) {
            kz[1] = wrapi(k2 + 1, K.n2, K.p2);
            wz[0] = wz[1] = (T)0.5;
        }
        // KIND 0: coarse columns and rows I-1, I, I+1; KIND 1: I, I+1
        constexpr int W = KIND == 0 ? 3 : 2;
        int cx[W], cy[W];
        bool okx[W], oky[W];
#pragma unroll
        for (int o = 0; o < W; o++) {
            const int xx = wrapi(I + o - (KIND == 0 ? 1 : 0), K.n0, K.p0), yy = wrapi(J + o - (KIND == 0 ? 1 : 0), K.n1, K.p1);
            okx[o] = xx >= 0;
            oky[o] = yy >= 0;
            cx[o] = col(K, xx < 0 ? I : xx);
            cy[o] = ((yy < 0 ? J : yy) + 1) * K.RS;
        }
        T e[4] = {0, 0, 0, 0};  // [b][a]
#pragma unroll
        for (int c = 0; c < 2; c++) {
            if (c == 1 && wz[1] == 0) break;
            const int rk = fdiv(kz[c], K.inv_q);
            const T *pl = cl_map(C.sm, rk) + K.ox + (kz[c] - rk * K.q + 1) * K.PX;
            T v[W][W];
#pragma unroll
            for (int b = 0; b < W; b++)
#pragma unroll
                for (int a = 0; a < W; a++) v[b][a] = pl[cy[b] + cx[a]];
#pragma unroll
            for (int b = 0; b < 2; b++)
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    T &ee = e[2 * b + a];
                    if (KIND == 0) {
                        // odd points lean on the next coarse cell, even on the
                        // previous; without it the near cell counts fully
                        const int na = a ? 2 : 0, nb = b ? 2 : 0;
                        const T wx[2] = {okx[na] ? (T)0.75 : (T)1, okx[na] ? (T)0.25 : (T)0};
                        const T wy[2] = {oky[nb] ? (T)0.75 : (T)1, oky[nb] ? (T)0.25 : (T)0};
                        ee += wx[0] * wy[0] * wz[c] * v[1][1];
                        ee += wx[1] * wy[0] * wz[c] * v[1][na];
                        ee += wx[0] * wy[1] * wz[c] * v[nb][1];
                        ee += wx[1] * wy[1] * wz[c] * v[nb][na];
                    } else {
                        const T wx = a ? (T)0.5 : (T)1, wy = b ? (T)0.5 : (T)1, w = wx * wy * wz[c];
                        ee += w * v[0][0];
                        if (a) ee += w * v[0][1];
                        if (b) ee += w * v[1][0];
                        if (a && b) ee += w * v[1][1];
                    }
                }
        }
#pragma unroll
        for (int b = 0; b < 2; b++)
#pragma unroll
            for (int a = 0; a < 2; a++) {
                const int i = 2 * I + a, j = 2 * J + b;
                if (i >= V.n0 || j >= V.n1) continue;
                const int o = (j + 1) * V.RS + I + (a ? 1 : V.H);
                const T xo = C.sm[V.ox + kl * V.PX + o];
                put_x<T, true>(C, V, i, j, kl, o, xo + e[2 * b + a], -1);
            }
    }
}

// coarsest level: x = B r, one warp per row of the dense inverse, each row
// summed in the order of body_coarse_dense; a warp's rows run together so
// that their loads overlap
template <typename T>
__device__ __forceinline__ void dense_level(const slab_ctx<T> &C, const slab_args &S, const slab_level &L,
                                            const double *__restrict__ B) {
    const double *rs = reinterpret_cast<const double *>(reinterpret_cast<const unsigned char *>(C.sm) + S.dense_off);
    const int np = L.n0 * L.n1 * L.n2;
    const int warp = C.tid >> 5, lane = C.tid & 31, nw = kSlabThreads / 32 * S.csize;
    constexpr int R = 3;
    for (int row0 = C.rank * (kSlabThreads / 32) + warp; row0 < np; row0 += R * nw) {
        double acc[R];
        const double *b[R];
#pragma unroll
        for (int q = 0; q < R; q++) {
            acc[q] = 0;
            const int row = row0 + q * nw;
            b[q] = B + (size_t)(row < np ? row : np - 1) * np;
        }
#pragma unroll 8
        for (int c = lane; c < np; c += 32) {
            const double r = rs[c];
#pragma unroll
            for (int q = 0; q < R; q++) acc[q] += b[q][c] * r;
        }
#pragma unroll
        for (int q = 0; q < R; q++) {
            for (int o = 16; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
            const int row = row0 + q * nw;
            if (lane == 0 && row < np) {
                const int yz = fdiv(row, L.inv_n0), i = row - yz * L.n0;
                const int k = fdiv(yz, L.inv_n1), j = yz - k * L.n1;
                const int rk = fdiv(k, L.inv_q);
                cl_map(C.sm, rk)[L.ox + (k - rk * L.q + 1) * L.PX + (j + 1) * L.RS + col(L, i)] = (T)acc[q];
            }
        }
    }
}

template <typename T, int KIND, bool VD>
__device__ __forceinline__ void slab_cycle(const pmg_args &A, const slab_args &S, unsigned char *raw) {
    slab_ctx<T> C;
    C.sm = reinterpret_cast<T *>(raw);
    C.rank = (int)cl_rank();
    C.tid = threadIdx.x;
    C.bar = reinterpret_cast<uint64_t *>(raw + S.bar_off);
    C.failed = reinterpret_cast<int *>(raw + S.bar_off + 2 * sizeof(uint64_t));
    const int nl = S.nlev;
    int use = 0;
    if (C.tid == 0) {
        halo_init(C.bar);
        halo_init(C.bar + 1);
        halo_init_fence();
        *C.failed = 0;
    }
    slab_pass *pass = reinterpret_cast<slab_pass *>(raw + S.pass_off);
    constexpr int nc = KIND == 1 ? 4 : 2;
    for (int t = C.tid; t < 4 * (nl - 1); t += kSlabThreads)
        if ((t & 3) < nc) make_pass<T, KIND>(S.lv[t >> 2], C.rank, t & 3, pass + t);
    // x and 1/rho start at zero everywhere (ghosts beyond walls stay zero)
    for (int t = C.tid; t < S.zero_elems; t += kSlabThreads) C.sm[t] = 0;
    __syncthreads();
    {
        const slab_level &L = S.lv[0];
        const pmg_level &G = A.lv[S.l0];
        const T *gr = LR<T>(G), *gx = LX<T>(G);
        const int np = nplanes(L, C.rank), k0 = C.rank * L.q;
        const int tot = L.n0 * L.n1 * np;
        const size_t g0 = (size_t)L.n0 * L.n1 * k0;
        for (int t = C.tid; t < tot; t += kSlabThreads) {
            const int row = fdiv(t, L.inv_n0), i = t - row * L.n0;
            const int kl = fdiv(row, L.inv_n1), j = row - kl * L.n1;
            C.sm[L.orr + kl * L.PR + j * L.RS + col(L, i)] = gr[g0 + t];
        }
        const slab_view<T> V = view_of(C, L);
        if (S.load_x && np > 0)
            for (int kl = -1; kl <= np; kl++) {
                const int k = wrapi(k0 + kl, L.n2, L.p2);
                if (k < 0) continue;
                const T *g = gx + (size_t)L.n0 * L.n1 * k;
                for (int t = C.tid; t < L.n0 * L.n1; t += kSlabThreads) {
                    const int j = fdiv(t, L.inv_n0), i = t - j * L.n0;
                    put_images(V, C.sm + (V.ox + kl * V.PX), i, j, (j + 1) * V.RS + col(L, i), g[t]);
                }
            }
    }
    if (VD)
        for (int l = 0; l < nl - 1; l++) {
            // cells of the slab's planes and one layer around, with images
            const slab_level &L = S.lv[l];
            const T *__restrict__ ri = LRI<T>(A.lv[S.l0 + l]);
            const int c0 = KIND == 1 && !L.p0 ? L.n0 - 1 : L.n0, c1 = KIND == 1 && !L.p1 ? L.n1 - 1 : L.n1,
                      c2 = KIND == 1 && !L.p2 ? L.n2 - 1 : L.n2;
            const int np = nplanes(L, C.rank), k0 = C.rank * L.q;
            if (np == 0) continue;
            const int wx = L.n0 + 2, wy = L.n1 + 2;
#pragma unroll 4
            for (int t = C.tid; t < wx * wy * (np + 2); t += kSlabThreads) {
                const int row = fdiv(t, L.inv_w0), ii = t - row * wx;
                const int kl = fdiv(row, L.inv_w1), jj = row - kl * wy;
                const int i = wrapi(ii - 1, c0, L.p0), j = wrapi(jj - 1, c1, L.p1), k = wrapi(k0 + kl - 1, c2, L.p2);
                // (a node may have an index past the last cell of a walled axis)
                const bool ok = (i | j | k) >= 0;
                const T v = ri[ok ? i + c0 * (j + (size_t)c1 * k) : 0];
                C.sm[L.oi + kl * L.PX + jj * L.RS + col(L, ii - 1)] = ok ? v : (T)0;
            }
        }
    cl_barrier();
    for (int l = 0; l < nl - 1; l++) {
        const slab_level &L = S.lv[l];
        const slab_view<T> V = view_of(C, L);
        smooth_level<T, KIND, VD>(C, V, A.v_down, pass + 4 * l, use);
        for (int c = 0; c < nc; c++) colour_pass<T, KIND, VD, 1>(C, pass[4 * l + c], V, c, -1);
        cl_barrier();
        restrict_level<T, KIND>(C, S, L, S.lv[l + 1], l + 1 == nl - 1);
        cl_barrier();
    }
    dense_level(C, S, S.lv[nl - 1], A.dense);
    cl_barrier();
    for (int l = nl - 2; l >= 0; l--) {
        const slab_level &L = S.lv[l];
        const slab_view<T> V = view_of(C, L);
        prolong_level<T, KIND>(C, L, S.lv[l + 1], V);
        cl_barrier();
        smooth_level<T, KIND, VD>(C, V, A.v_up, pass + 4 * l, use);
        cl_barrier();  // the next finer level reads x across slabs; no CTA leaves with sends under way
    }
    {
        const slab_level &L = S.lv[0];
        T *gx = LX<T>(A.lv[S.l0]);
        const int np = nplanes(L, C.rank);
        const int tot = L.n0 * L.n1 * np;
        const size_t g0 = (size_t)L.n0 * L.n1 * C.rank * L.q;
        for (int t = C.tid; t < tot; t += kSlabThreads) {
            const int row = fdiv(t, L.inv_n0), i = t - row * L.n0;
            const int kl = fdiv(row, L.inv_n1), j = row - kl * L.n1;
            const T v = C.sm[L.ox + (kl + 1) * L.PX + (j + 1) * L.RS + col(L, i)];
            gx[g0 + t] = *C.failed ? (T)NAN : v;
        }
    }
    // a wait that gave up: the solve's control reports it, and this CTA stays
    // until what is still under way to its shared memory has arrived
    if (*C.failed) {
        if (C.tid == 0) *A.gave_up = 1;
        cl_linger();
    }
}

// Layout of levels l0 .. coarsest over csize CTAs; bytes per CTA, or 0 when a
// count exceeds what the index arithmetic covers
inline size_t slab_layout(const std::vector<mg_level> &lv, int l0, int csize, bool f64, bool vd, bool load_x, slab_args *out) {
    slab_args S;
    memset(&S, 0, sizeof(S));
    S.l0 = l0;
    S.nlev = (int)lv.size() - l0;
    S.csize = csize;
    S.load_x = load_x;
    if (S.nlev < 2 || S.nlev > kMaxLev) return 0;
    size_t off = 0, res = 0;
    auto inv = [](int d) { return (unsigned)((0x80000000ull + d - 1) / d); };
    for (int pass = 0; pass < 2; pass++)  // x and 1/rho first (zeroed), then r
        for (int l = 0; l < S.nlev; l++) {
            slab_level &L = S.lv[l];
            const mg_level &M = lv[l0 + l];
            if (pass == 0) {
                L.n0 = M.n[0], L.n1 = M.n[1], L.n2 = M.n[2];
                L.p0 = M.prd[0], L.p1 = M.prd[1], L.p2 = M.prd[2];
                L.q = (L.n2 + csize - 1) / csize;
                L.H = (L.n0 + 3) / 2;
                L.RS = 2 * L.H;
                L.PX = (L.n1 + 2) * L.RS;
                L.PR = L.n1 * L.RS;
                L.inv_n0 = inv(L.n0), L.inv_n1 = inv(L.n1), L.inv_q = inv(L.q);
                L.inv_w0 = inv(L.n0 + 2), L.inv_w1 = inv(L.n1 + 2), L.inv_half = inv((L.n0 + 1) / 2);
                // columns of each parity: all, and those off the rim
                auto cols = [&](int n, int c) {
                    slab_col q;
                    q.n = (n - c + 1) / 2;
                    q.lo = c == 0 ? 1 : 0;
                    q.in = q.n - q.lo - (((n - 1) & 1) == c && n > 1 ? 1 : 0);
                    if (q.in < 0) q.in = 0;
                    q.inv_in = inv(q.in > 0 ? q.in : 1);
                    return q;
                };
                for (int c = 0; c < 2; c++) L.cx[c] = cols(L.n0, c), L.cy[c] = cols(L.n1, c);
                for (int c = 0; c < 4; c++) {
                    const slab_col &X = L.cx[c & 1], &Y = L.cy[c >> 1];
                    const int in = X.in * Y.in, rim = X.n * Y.n - in;
                    L.inv_in[c] = inv(in > 0 ? in : 1);
                    L.inv_rim[c] = inv(rim > 0 ? rim : 1);
                }
                // fdiv's range
                const long long plane = (long long)(L.n0 + 2) * (L.n1 + 2);
                if (plane * (L.q + 2) > (1 << 16) || plane > (1 << 14)) return 0;
                L.ox = (int)off;
                off += (size_t)(L.q + 2) * L.PX;
                if (vd && l < S.nlev - 1) {
                    L.oi = (int)off;
                    off += (size_t)(L.q + 2) * L.PX;
                }
            } else {
                L.orr = (int)off;
                off += (size_t)L.q * L.PR;
                if (l < S.nlev - 1) res = std::max(res, (size_t)L.q * L.PR);
            }
            if (pass == 0 && l == S.nlev - 1) S.zero_elems = (int)off;
        }
    for (int l = 0; l < S.nlev; l++) S.lv[l].os = (int)off;
    off += res;
    const size_t elem = f64 ? 8 : 4;
    size_t bytes = (off * elem + 15) & ~(size_t)15;
    S.dense_off = (int)bytes;
    bytes += lv.back().npts() * sizeof(double);
    S.bar_off = (int)bytes;
    bytes += 2 * sizeof(uint64_t) + 16;
    bytes = (bytes + 15) & ~(size_t)15;
    S.pass_off = (int)bytes;
    bytes += 4 * (S.nlev - 1) * sizeof(slab_pass);
    if (out) *out = S;
    return bytes;
}

}  // namespace rmt3d
