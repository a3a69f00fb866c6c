// Multigrid operator helpers of the V-cycle kernels (k_mg.cu): rediscretised
// MAC 7-point and FEM Q1 27-point stencils with the boundary rules of
// stencil_set::set_partials (Utilities/mg_probs.hh:281-343), and the phases of
// the one-block coarse sub-cycle.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace rmt3d {

struct lvl_dev {
    int n0, n1, n2;
    int p0, p1, p2;
};

__host__ __device__ __forceinline__ int wrapi(int v, int n, int prd) {
    if (v < 0) return prd ? v + n : -1;
    if (v >= n) return prd ? v - n : -1;
    return v;
}

// v / num for num in {1, 2, 4, 8} as an exact power-of-two scaling (the same
// bits as the division, without its instruction sequence)
template <typename T>
__device__ __forceinline__ T div_pow2(T v, int num) {
    return num == 1 ? v : num == 2 ? v * (T)0.5 : num == 4 ? v * (T)0.25 : num == 8 ? v * (T)0.125 : v / (T)num;
}

// ---- operator application -------------------------------------------------
// The sum of the off-diagonal terms of one row and its diagonal.  Interior
// and rim points load the same neighbours (a missing one's place is taken by
// any stored value), so a warp that holds the end of a row loads once: rim
// points, about one in every warp of a 64^3 level, then only sum in another
// way -- term by term, missing neighbours with coefficient zero, whose terms
// leave the sum's bits alone.

// offsets to the lower and upper neighbour along an axis of n >= 2 points
// (stride st): the image across a periodic seam; beyond a wall the neighbour
// on the other side stands in (never a point of the same colour, so nothing
// that a colour pass is writing is read)
__device__ __forceinline__ int nb_lo(int c, int n, int prd, int st) { return c > 0 ? -st : (prd ? (n - 1) * st : st); }
__device__ __forceinline__ int nb_hi(int c, int n, int prd, int st) { return c < n - 1 ? st : (prd ? (1 - n) * st : -st); }

template <typename T>
__device__ __forceinline__ T mac_sum(const lvl_dev &L, int i, int j, int k, T xm, T xp, T ym, T yp, T zm, T zp, T &diag) {
    if (i > 0 && i < L.n0 - 1 && j > 0 && j < L.n1 - 1 && k > 0 && k < L.n2 - 1) {
        diag = (T)-6;
        return ((xm + xp) + (ym + yp)) + (zm + zp);
    }
    const bool a0 = i == 0 && !L.p0, a1 = i == L.n0 - 1 && !L.p0, b0 = j == 0 && !L.p1, b1 = j == L.n1 - 1 && !L.p1,
               c0 = k == 0 && !L.p2, c1 = k == L.n2 - 1 && !L.p2;
    T s = 0;
    s += a0 ? (T)0 : xm;
    s += a1 ? (T)0 : xp;
    s += b0 ? (T)0 : ym;
    s += b1 ? (T)0 : yp;
    s += c0 ? (T)0 : zm;
    s += c1 ? (T)0 : zp;
    diag = (T)(-6 + (int)a0 + (int)a1 + (int)b0 + (int)b1 + (int)c0 + (int)c1);
    return s;
}

template <typename T>
__device__ __forceinline__ T mac_offdiag(const lvl_dev L, const T *__restrict__ x, int i, int j, int k, T &diag) {
    const int sy = L.n0, sz = L.n0 * L.n1;
    const T *c = x + i + sy * j + sz * k;
    T xm = c[nb_lo(i, L.n0, L.p0, 1)], xp = c[nb_hi(i, L.n0, L.p0, 1)];
    T ym = c[nb_lo(j, L.n1, L.p1, sy)], yp = c[nb_hi(j, L.n1, L.p1, sy)];
    T zm = c[nb_lo(k, L.n2, L.p2, sz)], zp = c[nb_hi(k, L.n2, L.p2, sz)];
    return mac_sum(L, i, j, k, xm, xp, ym, yp, zm, zp, diag);
}

// the constant-density FEM sum of a node on the rim of the level, term by
// term: a.., b.., d.. the planes below, of and above the node, digits x and y
template <typename T>
__device__ __forceinline__ T fem_rim_sum(const lvl_dev &L, int i, int j, int k, T a00, T a10, T a20, T a01, T a21, T a02,
                                         T a12, T a22, T b00, T b20, T b02, T b22, T d00, T d10, T d20, T d01, T d21,
                                         T d02, T d12, T d22, T &diag) {
    // 1 where the neighbour on that side exists; an entry is halved once per
    // wall plane the node lies on along an axis it does not move along
    const bool wx = !L.p0 && (i == 0 || i == L.n0 - 1), wy = !L.p1 && (j == 0 || j == L.n1 - 1),
               wz = !L.p2 && (k == 0 || k == L.n2 - 1);
    const T x0 = !L.p0 && i == 0 ? (T)0 : (T)1, x1 = !L.p0 && i == L.n0 - 1 ? (T)0 : (T)1;
    const T v0 = !L.p1 && j == 0 ? (T)0 : (T)1, v1 = !L.p1 && j == L.n1 - 1 ? (T)0 : (T)1;
    const T z0 = !L.p2 && k == 0 ? (T)0 : (T)1, z1 = !L.p2 && k == L.n2 - 1 ? (T)0 : (T)1;
    const T ex = wx ? (T)-1 : (T)-2, ey = wy ? (T)-1 : (T)-2, ez = wz ? (T)-1 : (T)-2;
    const T p00 = x0 * v0, p20 = x1 * v0, p02 = x0 * v1, p22 = x1 * v1;
    T s = 0;
    s += -(p00 * z0) * a00;
    s += ex * (v0 * z0) * a10;
    s += -(p20 * z0) * a20;
    s += ey * (x0 * z0) * a01;
    s += ey * (x1 * z0) * a21;
    s += -(p02 * z0) * a02;
    s += ex * (v1 * z0) * a12;
    s += -(p22 * z0) * a22;
    s += ez * p00 * b00;
    s += ez * p20 * b20;
    s += ez * p02 * b02;
    s += ez * p22 * b22;
    s += -(p00 * z1) * d00;
    s += ex * (v0 * z1) * d10;
    s += -(p20 * z1) * d20;
    s += ey * (x0 * z1) * d01;
    s += ey * (x1 * z1) * d21;
    s += -(p02 * z1) * d02;
    s += ex * (v1 * z1) * d12;
    s += -(p22 * z1) * d22;
    diag = (T)(32 >> ((int)wx + (int)wy + (int)wz));
    return s;
}

template <typename T>
__device__ __forceinline__ T fem_offdiag(const lvl_dev L, const T *__restrict__ x, int i, int j, int k, T &diag) {
    // edges -2, corners -1, faces 0
    const int sy = L.n0, sz = L.n0 * L.n1;
    const int xl = nb_lo(i, L.n0, L.p0, 1), xh = nb_hi(i, L.n0, L.p0, 1);
    const T *c = x + i + sy * j + sz * k;
    const T *y0 = c + nb_lo(j, L.n1, L.p1, sy), *y2 = c + nb_hi(j, L.n1, L.p1, sy);
    const int zl = nb_lo(k, L.n2, L.p2, sz), zh = nb_hi(k, L.n2, L.p2, sz);
    const T a00 = y0[zl + xl], a10 = y0[zl], a20 = y0[zl + xh], a01 = c[zl + xl], a21 = c[zl + xh], a02 = y2[zl + xl],
            a12 = y2[zl], a22 = y2[zl + xh];
    const T b00 = y0[xl], b20 = y0[xh], b02 = y2[xl], b22 = y2[xh];
    const T d00 = y0[zh + xl], d10 = y0[zh], d20 = y0[zh + xh], d01 = c[zh + xl], d21 = c[zh + xh], d02 = y2[zh + xl],
            d12 = y2[zh], d22 = y2[zh + xh];
    if (i > 0 && i < L.n0 - 1 && j > 0 && j < L.n1 - 1 && k > 0 && k < L.n2 - 1) {
        T e = (b00 + b20) + (b02 + b22);
        e += (a01 + a21) + (a10 + a12);
        e += (d01 + d21) + (d10 + d12);
        T q = (a00 + a20) + (a02 + a22);
        q += (d00 + d20) + (d02 + d22);
        diag = (T)32;
        return (T)-2 * e - q;
    }
    return fem_rim_sum(L, i, j, k, a00, a10, a20, a01, a21, a02, a12, a22, b00, b20, b02, b22, d00, d10, d20, d01, d21,
                       d02, d12, d22, diag);
}

// walled axes x and y on whose end planes a FEM node lies
__device__ __forceinline__ int fem_walls(const lvl_dev &L, int i, int j) {
    return (!L.p0 && (i == 0 || i == L.n0 - 1)) + (!L.p1 && (j == 0 || j == L.n1 - 1));
}

// 1 / diag of the constant-density FEM stencil at node (i, j, k).  diag is
// 32 / 2^h, h the number of walled axes on whose end planes the node lies,
// so the reciprocal 2^h / 32 is exact and (r - s) times it has the same bits
// as (r - s) / diag, without a division's instruction sequence.
template <typename T>
__device__ __forceinline__ T fem_inv_diag(const lvl_dev L, int i, int j, int k) {
    const int h = (!L.p0 && (i == 0 || i == L.n0 - 1)) + (!L.p1 && (j == 0 || j == L.n1 - 1)) +
                  (!L.p2 && (k == 0 || k == L.n2 - 1));
    return (T)(1 << h) * (T)0.03125;
}

// ---- variable density (VAR_DEN) ---------------------------------------------
// ri: 1/rho per cell of the level (cell-centred, MAC level dimensions; for a
// FEM level with n nodes per axis there are n-1 cells on a walled axis and n
// on a periodic one).  Coarse levels carry the mean of their 8 children.

// var_den_mac::set_stencils (Utilities/mg_probs.cc:196-308): each face
// coefficient is the mean of 1/rho of the two cells it joins; the centre is
// the (Neumann-fixed) centre entry times the mean of the face coefficients,
// accumulated direction by direction as the reference does.
template <typename T>
__device__ __forceinline__ T mac_offdiag_vd(const lvl_dev L, const T *__restrict__ x, const T *__restrict__ ri, int i,
                                            int j, int k, T &diag) {
    const int sy = L.n0, sz = L.n0 * L.n1, base = i + sy * j + sz * k;
    const T *c = x + base, *q = ri + base;
    const int xl = nb_lo(i, L.n0, L.p0, 1), xh = nb_hi(i, L.n0, L.p0, 1), yl = nb_lo(j, L.n1, L.p1, sy),
              yh = nb_hi(j, L.n1, L.p1, sy), zl = nb_lo(k, L.n2, L.p2, sz), zh = nb_hi(k, L.n2, L.p2, sz);
    const T rc = q[0];
    const bool a0 = i > 0 || L.p0, a1 = i < L.n0 - 1 || L.p0, b0 = j > 0 || L.p1, b1 = j < L.n1 - 1 || L.p1,
               c0 = k > 0 || L.p2, c1 = k < L.n2 - 1 || L.p2;
    const T ax1 = a0 ? (T)0.5 * (q[xl] + rc) : (T)0, ax2 = a1 ? (T)0.5 * (rc + q[xh]) : (T)0;
    const T ay1 = b0 ? (T)0.5 * (q[yl] + rc) : (T)0, ay2 = b1 ? (T)0.5 * (rc + q[yh]) : (T)0;
    const T az1 = c0 ? (T)0.5 * (q[zl] + rc) : (T)0, az2 = c1 ? (T)0.5 * (rc + q[zh]) : (T)0;
    T s = 0, csum = 0;
    s += ax1 * c[xl] + ax2 * c[xh];
    csum += ax1 + ax2;
    s += ay1 * c[yl] + ay2 * c[yh];
    csum += ay1 + ay2;
    s += az1 * c[zl] + az2 * c[zh];
    csum += az1 + az2;
    const int cnt = (int)a0 + (int)a1 + (int)b0 + (int)b1 + (int)c0 + (int)c1;
    diag = (T)(-cnt) * (csum / (T)cnt);
    return s;
}

// var_den_fem::set_stencils (Utilities/mg_probs.cc:97-150): every entry of the
// (boundary-halved) Q1 stencil is scaled by the mean of 1/rho over the cells
// adjacent to both the node and that neighbour -- 1 cell for a corner
// neighbour, 2 for an edge neighbour, all (up to 8) for the centre -- summed
// in the reference's cell order.  With a missing cell's 1/rho as zero that is
// -v for a corner, -(va + vb) for an edge (twice the mean of two cells, or
// once the one cell that a wall leaves, with the entry halved) and 4 times
// the sum for the centre, each exactly; a missing neighbour has no cells.
template <typename T>
__device__ __forceinline__ T fem_offdiag_vd(const lvl_dev L, const T *__restrict__ x, const T *__restrict__ ri, int i,
                                            int j, int k, T &diag) {
    const int sy = L.n0, sz = L.n0 * L.n1;
    const int ncx = L.p0 ? L.n0 : L.n0 - 1, ncy = L.p1 ? L.n1 : L.n1 - 1, ncz = L.p2 ? L.n2 : L.n2 - 1;
    // cells below and above the node on each axis, -1: none
    const int i0 = i > 0 ? i - 1 : (L.p0 ? ncx - 1 : -1), i1 = i < ncx ? i : -1;
    const int j0 = j > 0 ? j - 1 : (L.p1 ? ncy - 1 : -1), j1 = j < ncy ? j : -1;
    const int k0 = k > 0 ? k - 1 : (L.p2 ? ncz - 1 : -1), k1 = k < ncz ? k : -1;
    auto cell = [&](int a, int b, int c) -> T { return (a | b | c) >= 0 ? ri[a + ncx * (b + ncy * c)] : (T)0; };
    const T u00 = cell(i0, j0, k0), u10 = cell(i1, j0, k0), u01 = cell(i0, j1, k0), u11 = cell(i1, j1, k0);
    const T v00 = cell(i0, j0, k1), v10 = cell(i1, j0, k1), v01 = cell(i0, j1, k1), v11 = cell(i1, j1, k1);
    const int xl = nb_lo(i, L.n0, L.p0, 1), xh = nb_hi(i, L.n0, L.p0, 1);
    const T *c = x + i + sy * j + sz * k;
    const T *y0 = c + nb_lo(j, L.n1, L.p1, sy), *y2 = c + nb_hi(j, L.n1, L.p1, sy);
    const int zl = nb_lo(k, L.n2, L.p2, sz), zh = nb_hi(k, L.n2, L.p2, sz);
    T s = 0;
    s += -u00 * y0[zl + xl];
    s += -(u00 + u10) * y0[zl];
    s += -u10 * y0[zl + xh];
    s += -(u00 + u01) * c[zl + xl];
    s += -(u10 + u11) * c[zl + xh];
    s += -u01 * y2[zl + xl];
    s += -(u01 + u11) * y2[zl];
    s += -u11 * y2[zl + xh];
    s += -(u00 + v00) * y0[xl];
    s += -(u10 + v10) * y0[xh];
    s += -(u01 + v01) * y2[xl];
    s += -(u11 + v11) * y2[xh];
    s += -v00 * y0[zh + xl];
    s += -(v00 + v10) * y0[zh];
    s += -v10 * y0[zh + xh];
    s += -(v00 + v01) * c[zh + xl];
    s += -(v10 + v11) * c[zh + xh];
    s += -v01 * y2[zh + xl];
    s += -(v01 + v11) * y2[zh];
    s += -v11 * y2[zh + xh];
    T c8 = 0;
    c8 += u00;
    c8 += u10;
    c8 += u01;
    c8 += u11;
    c8 += v00;
    c8 += v10;
    c8 += v01;
    c8 += v11;
    diag = (T)4 * c8;
    return s;
}

template <typename T>
__device__ __forceinline__ T op_offdiag(int kind, const lvl_dev L, const T *__restrict__ x, const T *__restrict__ ri,
                                        int i, int j, int k, T &diag) {
    if (ri) return kind == 0 ? mac_offdiag_vd(L, x, ri, i, j, k, diag) : fem_offdiag_vd(L, x, ri, i, j, k, diag);
    return kind == 0 ? mac_offdiag(L, x, i, j, k, diag) : fem_offdiag(L, x, i, j, k, diag);
}

constexpr int kMaxLev = 12;
constexpr int kDensePts = 1000;  // coarsening stops at the first level with at most this many points
constexpr int kDenseMax = 1024;  // largest level solved by a dense inverse
constexpr int kThreads = 256;

struct pmg_level {
    int n[3];
    int prd[3];
    double *x, *r, *res;
    float *xs, *rs, *ress;
    const double *ri;  // variable density: 1/rho per cell (null: constant)
    const float *ris;
};

struct pmg_args {
    int kind;  // 0 MAC, 1 FEM
    int nlev;
    pmg_level lv[kMaxLev];
    const double *dense;  // inverse of the coarsest operator, or null
    int v_up, v_down;
    int *gave_up;  // the solve's mg_ctl::gave_up (the shared-memory V-cycle sets it)
};

// the columns (or rows) of one parity: their number, the number off the rim
// of the plane, whether the first one lies on the rim
struct slab_col {
    int n, in, lo;
    unsigned inv_in;
};
// One level of a V-cycle part held in shared memory, cut into slabs of q
// planes (k_mgs.cu).  Offsets and strides in elements of a CTA's arrays.
struct slab_level {
    int n0, n1, n2, p0, p1, p2;
    int q;              // planes per CTA
    int H, RS, PX, PR;  // half row, row, plane of x (with ghosts), plane of r
    int ox, orr, os, oi;  // x, r, residual, 1/rho
    // reciprocals for index division
    unsigned inv_n0, inv_n1, inv_q, inv_w0, inv_w1, inv_half, inv_in[4], inv_rim[4];
    slab_col cx[2], cy[2];  // FEM: the colours' columns and rows
};
struct slab_args {
    int l0, nlev, csize, load_x;
    int zero_elems;  // x and 1/rho arrays, zeroed at the start
    int dense_off;   // bytes: the coarsest right-hand side in FP64
    int bar_off;     // bytes: two mbarriers and a flag
    int pass_off;    // bytes: the passes' tables
    slab_level lv[kMaxLev];
};

__device__ __forceinline__ lvl_dev ldev(const pmg_level &L) {
    return lvl_dev{L.n[0], L.n[1], L.n[2], L.prd[0], L.prd[1], L.prd[2]};
}

// ---- one phase over a level, for the points [t0, total) with stride ts ----
template <typename T>
__device__ void ph_smooth_colour(int kind, const lvl_dev L, T *x, const T *r, const T *ri, int colour, int t0, int ts) {
    if (kind == 0) {
        const int h = (L.n0 + 1) / 2;
        const int tot = h * L.n1 * L.n2;
        for (int t = t0; t < tot; t += ts) {
            int hi = t % h, j = (t / h) % L.n1, k = t / (h * L.n1);
            int i = 2 * hi + ((j + k + colour) & 1);
            if (i >= L.n0) continue;
            T diag;
            T s = op_offdiag<T>(0, L, x, ri, i, j, k, diag);
            int id = i + L.n0 * (j + L.n1 * k);
            x[id] = (r[id] - s) / diag;
        }
    } else {
        const int ha = (L.n0 + 1) / 2, hb = (L.n1 + 1) / 2;
        const int tot = ha * hb * L.n2;
        for (int t = t0; t < tot; t += ts) {
            int a = t % ha, b = (t / ha) % hb, k = t / (ha * hb);
            int i = 2 * a + (colour & 1), j = 2 * b + ((colour >> 1) & 1);
            if (i >= L.n0 || j >= L.n1) continue;
            T diag;
            T s = op_offdiag<T>(1, L, x, ri, i, j, k, diag);
            int id = i + L.n0 * (j + L.n1 * k);
            x[id] = (r[id] - s) / diag;
        }
    }
}

template <typename T>
__device__ double ph_resid(int kind, const lvl_dev L, const T *x, const T *r, T *res, const T *ri, int t0, int ts) {
    const int tot = L.n0 * L.n1 * L.n2;
    double mx = 0;
    for (int t = t0; t < tot; t += ts) {
        int i = t % L.n0, j = (t / L.n0) % L.n1, k = t / (L.n0 * L.n1);
        T diag;
        T s = op_offdiag<T>(kind, L, x, ri, i, j, k, diag);
        T v = r[t] - s - diag * x[t];
        if (res) res[t] = v;
        double a = fabs((double)v);
        if (a != a || a > mx) mx = a;  // NaN sticks
    }
    return mx;
}

template <typename T>
__device__ void ph_restrict(int kind, const lvl_dev F, const lvl_dev C, const T *res, T *rc, T *xc, int t0, int ts) {
    const int tot = C.n0 * C.n1 * C.n2;
    for (int t = t0; t < tot; t += ts) {
        int I = t % C.n0, J = (t / C.n0) % C.n1, K = t / (C.n0 * C.n1);
        T s = 0;
        if (kind == 0) {
            for (int c = 0; c < 2; c++)
                for (int b = 0; b < 2; b++)
                    for (int a = 0; a < 2; a++) s += res[(2 * I + a) + F.n0 * ((2 * J + b) + F.n1 * (2 * K + c))];
        } else {
            const int nf[3] = {F.n0, F.n1, F.n2}, p[3] = {F.p0, F.p1, F.p2};
            const int cc[3] = {I, J, K};
            int idx[3][3];
            T w[3][3];
            for (int d = 0; d < 3; d++)
                for (int o = -1; o <= 1; o++) {
                    int v = wrapi(2 * cc[d] + o, nf[d], p[d]);
                    idx[d][o + 1] = v;
                    w[d][o + 1] = (v < 0) ? (T)0 : (o == 0 ? (T)1 : (T)0.5);
                }
            for (int oc = 0; oc < 3; oc++) {
                if (idx[2][oc] < 0) continue;
                for (int ob = 0; ob < 3; ob++) {
                    if (idx[1][ob] < 0) continue;
                    for (int oa = 0; oa < 3; oa++) {
                        if (idx[0][oa] < 0) continue;
                        s += w[0][oa] * w[1][ob] * w[2][oc] *
                             res[idx[0][oa] + F.n0 * (idx[1][ob] + F.n1 * idx[2][oc])];
                    }
                }
            }
        }
        rc[t] = (T)0.5 * s;
        xc[t] = 0;
    }
}

template <typename T>
__device__ void ph_prolong(int kind, const lvl_dev F, const lvl_dev C, T *x, const T *xc, int t0, int ts) {
    const int tot = F.n0 * F.n1 * F.n2;
    const int nc[3] = {C.n0, C.n1, C.n2}, p[3] = {C.p0, C.p1, C.p2};
    for (int t = t0; t < tot; t += ts) {
        int i = t % F.n0, j = (t / F.n0) % F.n1, k = t / (F.n0 * F.n1);
        const int f[3] = {i, j, k};
        int ci[3][2];
        T w[3][2];
        int cnt[3];
        for (int d = 0; d < 3; d++) {
            if (kind == 0) {
                int I = f[d] >> 1;
                int J = wrapi(I + ((f[d] & 1) ? 1 : -1), nc[d], p[d]);
                ci[d][0] = I;
                if (J < 0) {
                    w[d][0] = 1;
                    cnt[d] = 1;
                } else {
                    w[d][0] = (T)0.75;
                    ci[d][1] = J;
                    w[d][1] = (T)0.25;
                    cnt[d] = 2;
                }
            } else if ((f[d] & 1) == 0) {
                ci[d][0] = f[d] >> 1;
                w[d][0] = 1;
                cnt[d] = 1;
            } else {
                ci[d][0] = f[d] >> 1;
                ci[d][1] = wrapi((f[d] >> 1) + 1, nc[d], p[d]);
                w[d][0] = w[d][1] = (T)0.5;
                cnt[d] = 2;
            }
        }
        T e = 0;
        for (int c = 0; c < cnt[2]; c++)
            for (int b = 0; b < cnt[1]; b++)
                for (int a = 0; a < cnt[0]; a++)
                    e += w[0][a] * w[1][b] * w[2][c] * xc[ci[0][a] + C.n0 * (ci[1][b] + C.n1 * ci[2][c])];
        x[t] += e;
    }
}

template <typename T>
__device__ __forceinline__ void set_level_ptrs(pmg_level &L, T *x, T *r, T *res) {
    if constexpr (sizeof(T) == 8) {
        L.x = (double *)x;
        L.r = (double *)r;
        L.res = (double *)res;
    } else {
        L.xs = (float *)x;
        L.rs = (float *)r;
        L.ress = (float *)res;
    }
}

template <typename T>
__device__ __forceinline__ const T *LRI(const pmg_level &L) {
    if constexpr (sizeof(T) == 8) return (const T *)L.ri;
    else return (const T *)L.ris;
}

template <typename T>
__device__ __forceinline__ T *LX(const pmg_level &L) {
    if constexpr (sizeof(T) == 8) return (T *)L.x;
    else return (T *)L.xs;
}
template <typename T>
__device__ __forceinline__ T *LR(const pmg_level &L) {
    if constexpr (sizeof(T) == 8) return (T *)L.r;
    else return (T *)L.rs;
}
template <typename T>
__device__ __forceinline__ T *LS(const pmg_level &L) {
    if constexpr (sizeof(T) == 8) return (T *)L.res;
    else return (T *)L.ress;
}

// coarse levels cf..nlev-1 of one V-cycle inside the calling CTA
template <typename T>
__device__ void coarse_cycle(const pmg_args &A, int cf) {
    const int t0 = threadIdx.x, ts = blockDim.x;
    const int nc = A.kind == 0 ? 2 : 4;
    for (int l = cf; l < A.nlev - 1; l++) {
        const pmg_level &F = A.lv[l];
        for (int s = 0; s < A.v_down; s++)
            for (int c = 0; c < nc; c++) {
                ph_smooth_colour<T>(A.kind, ldev(F), LX<T>(F), LR<T>(F), LRI<T>(F), c, t0, ts);
                __syncthreads();
            }
        ph_resid<T>(A.kind, ldev(F), LX<T>(F), LR<T>(F), LS<T>(F), LRI<T>(F), t0, ts);
        __syncthreads();
        const pmg_level &C = A.lv[l + 1];
        ph_restrict<T>(A.kind, ldev(F), ldev(C), LS<T>(F), LR<T>(C), LX<T>(C), t0, ts);
        __syncthreads();
    }
    {  // coarsest level
        const pmg_level &L = A.lv[A.nlev - 1];
        const int np = L.n[0] * L.n[1] * L.n[2];
        T *x = LX<T>(L);
        const T *r = LR<T>(L);
        if (A.dense) {
            // one warp per row of the (row-major) inverse: coalesced reads
            const int warp = t0 >> 5, lane = t0 & 31, nw = ts >> 5;
            for (int row = warp; row < np; row += nw) {
                const double *b = A.dense + (size_t)row * np;
                double acc = 0;
                for (int c = lane; c < np; c += 32) acc += b[c] * (double)r[c];
                for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
                if (lane == 0) x[row] = (T)acc;
            }
            __syncthreads();
        } else {
            for (int p = t0; p < np; p += ts) x[p] = 0;
            __syncthreads();
            for (int s = 0; s < 80; s++)
                for (int c = 0; c < nc; c++) {
                    ph_smooth_colour<T>(A.kind, ldev(L), x, r, LRI<T>(L), c, t0, ts);
                    __syncthreads();
                }
        }
    }
    for (int l = A.nlev - 2; l >= cf; l--) {
        const pmg_level &F = A.lv[l];
        const pmg_level &C = A.lv[l + 1];
        ph_prolong<T>(A.kind, ldev(F), ldev(C), LX<T>(F), LX<T>(C), t0, ts);
        __syncthreads();
        for (int s = 0; s < A.v_up; s++)
            for (int c = 0; c < nc; c++) {
                ph_smooth_colour<T>(A.kind, ldev(F), LX<T>(F), LR<T>(F), LRI<T>(F), c, t0, ts);
                __syncthreads();
            }
    }
}

}  // namespace rmt3d
