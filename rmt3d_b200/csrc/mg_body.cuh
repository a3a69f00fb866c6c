// Bodies of the multigrid phase kernels, with the block coordinates passed
// in: the single-scene kernels (k_mg.cu) and the batched kernels that run a
// phase for every scene of a group in one launch (k_mgb.cu) call the same
// code, so a scene's solve gives the same bits alone and in a group.
#pragma once
#include <cuda_runtime.h>

#include "mg.h"
#include "mg_ops.cuh"

namespace rmt3d {

// A phase over a level runs blocks of 256 threads along each plane's points
// taken as one line (rows are 9 to 193 points: a block of whole rows would
// leave up to half its lanes idle), one plane per block row.  pt: the point's
// position on the line; split into row and column by the reciprocal
// inv = ceil(2^31 / n), exact while (2 pt + 1) n < 2^31.  With the rim in the
// interior's path (mg_ops.cuh), against 32 x 4 x 2 blocks and a separate rim
// path, on a B200: FP32 FEM colour pass of the 97^3 variable-density levels
// 9.2 -> 3.9 us, of 193^3 and 97^3 16.5 -> 11.8 us, FP64 of 65^3 4.9 -> 3.3 us.
__host__ __device__ __forceinline__ unsigned line_inv(int n) { return (unsigned)((0x80000000ull + n - 1) / n); }
__device__ __forceinline__ int line_row(int pt, unsigned inv) { return (int)__umulhi((unsigned)(2 * pt + 1), inv); }

// ---- smoothing -------------------------------------------------------------
template <typename T>
__device__ __forceinline__ void body_mac_rb(lvl_dev L, T *__restrict__ x, const T *__restrict__ r, int colour, const T *__restrict__ ri, unsigned inv, int pt, int k) {
    const int h = (L.n0 + 1) >> 1, j = line_row(pt, inv);
    const int i = 2 * (pt - j * h) + ((j + k + colour) & 1);
    if (j >= L.n1 || i >= L.n0) return;
    T diag;
    const T s = ri ? mac_offdiag_vd(L, x, ri, i, j, k, diag) : mac_offdiag(L, x, i, j, k, diag);
    const int id = i + L.n0 * (j + L.n1 * k);
    x[id] = (r[id] - s) / diag;
}

// A column of FEM nodes (i, j), planes k0 .. k1-1: emit(k, sum, diag, r,
// x) for each in turn (x only with OWN).  The eight neighbour columns slide through registers, nine loads a
// node instead of 21 (with variable density 13 instead of 29); sums and their
// order are those of fem_offdiag and fem_offdiag_vd.  No neighbour column is of
// the node's colour, so a pass may update the column as it goes; a plane's
// loads are issued ahead of the sums and the store of the plane before it.
template <typename T, bool VD, bool OWN, typename F>
__device__ __forceinline__ void fem_march(const lvl_dev &L, const T *x, const T *__restrict__ r, const T *__restrict__ ri, int i, int j, int k0,
                                          int k1, F emit) {
    const int sy = L.n0, sz = L.n0 * L.n1;
    const int xl = nb_lo(i, L.n0, L.p0, 1), xh = nb_hi(i, L.n0, L.p0, 1), yl = nb_lo(j, L.n1, L.p1, sy),
              yh = nb_hi(j, L.n1, L.p1, sy);
    // 0..3: (-,-) (+,-) (-,+) (+,+); 4..7: (-,0) (+,0) (0,-) (0,+)
    const int off[8] = {yl + xl, yl + xh, yh + xl, yh + xh, xl, xh, yl, yh};
    const T *c = x + i + sy * j + (size_t)sz * k0;
    const int zl = nb_lo(k0, L.n2, L.p2, sz);
    T w0[8], w1[8], w2[8], w3[8];
    const int zf = nb_hi(k0, L.n2, L.p2, sz);
#pragma unroll
    for (int q = 0; q < 8; q++) w0[q] = c[zl + off[q]], w1[q] = c[off[q]], w2[q] = c[zf + off[q]];
    T rv = r[i + sy * j + (size_t)sz * k0], xv = OWN ? c[0] : (T)0;
    const bool inside = i > 0 && i < L.n0 - 1 && j > 0 && j < L.n1 - 1;
    const int ncx = L.p0 ? L.n0 : L.n0 - 1, ncy = L.p1 ? L.n1 : L.n1 - 1, ncz = L.p2 ? L.n2 : L.n2 - 1;
    T u[4], v[4];
    int co[4];  // the column's cells of a layer, (y, x); -1: none
    if (VD) {
        const int i0 = i > 0 ? i - 1 : (L.p0 ? ncx - 1 : -1), i1 = i < ncx ? i : -1;
        const int j0 = j > 0 ? j - 1 : (L.p1 ? ncy - 1 : -1), j1 = j < ncy ? j : -1;
        co[0] = (i0 | j0) >= 0 ? i0 + ncx * j0 : -1;
        co[1] = (i1 | j0) >= 0 ? i1 + ncx * j0 : -1;
        co[2] = (i0 | j1) >= 0 ? i0 + ncx * j1 : -1;
        co[3] = (i1 | j1) >= 0 ? i1 + ncx * j1 : -1;
        const int kc = k0 > 0 ? k0 - 1 : (L.p2 ? ncz - 1 : -1);
#pragma unroll
        for (int q = 0; q < 4; q++) u[q] = (co[q] | kc) >= 0 ? ri[co[q] + (size_t)ncx * ncy * kc] : (T)0;
    }
    for (int k = k0; k < k1; k++, c += sz) {
        T rn = 0, xn = 0;
        if (k + 1 < k1) {
            const int zh = sz + nb_hi(k + 1, L.n2, L.p2, sz);
#pragma unroll
            for (int q = 0; q < 8; q++) w3[q] = c[zh + off[q]];
            rn = r[i + sy * j + (size_t)sz * (k + 1)];
            if (OWN) xn = c[sz];
        }
        T s, diag;
        if (VD) {
            const int kc = k < ncz ? k : -1;
#pragma unroll
            for (int q = 0; q < 4; q++) v[q] = (co[q] | kc) >= 0 ? ri[co[q] + (size_t)ncx * ncy * kc] : (T)0;
            s = 0;
            s += -u[0] * w0[0];
            s += -(u[0] + u[1]) * w0[6];
            s += -u[1] * w0[1];
            s += -(u[0] + u[2]) * w0[4];
            s += -(u[1] + u[3]) * w0[5];
            s += -u[2] * w0[2];
            s += -(u[2] + u[3]) * w0[7];
            s += -u[3] * w0[3];
            s += -(u[0] + v[0]) * w1[0];
            s += -(u[1] + v[1]) * w1[1];
            s += -(u[2] + v[2]) * w1[2];
            s += -(u[3] + v[3]) * w1[3];
            s += -v[0] * w2[0];
            s += -(v[0] + v[1]) * w2[6];
            s += -v[1] * w2[1];
            s += -(v[0] + v[2]) * w2[4];
            s += -(v[1] + v[3]) * w2[5];
            s += -v[2] * w2[2];
            s += -(v[2] + v[3]) * w2[7];
            s += -v[3] * w2[3];
            T c8 = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) c8 += u[q];
#pragma unroll
            for (int q = 0; q < 4; q++) c8 += v[q];
            diag = (T)4 * c8;
#pragma unroll
            for (int q = 0; q < 4; q++) u[q] = v[q];
        } else if (inside && k > 0 && k < L.n2 - 1) {
            T e = (w1[0] + w1[1]) + (w1[2] + w1[3]);
            e += (w0[4] + w0[5]) + (w0[6] + w0[7]);
            e += (w2[4] + w2[5]) + (w2[6] + w2[7]);
            T q = (w0[0] + w0[1]) + (w0[2] + w0[3]);
            q += (w2[0] + w2[1]) + (w2[2] + w2[3]);
            s = (T)-2 * e - q;
            diag = (T)32;
        } else {
            s = fem_rim_sum(L, i, j, k, w0[0], w0[6], w0[1], w0[4], w0[5], w0[2], w0[7], w0[3], w1[0], w1[1], w1[2],
                            w1[3], w2[0], w2[6], w2[1], w2[4], w2[5], w2[2], w2[7], w2[3], diag);
        }
        emit(k, s, diag, rv, xv);
#pragma unroll
        for (int q = 0; q < 8; q++) w0[q] = w1[q], w1[q] = w2[q], w2[q] = w3[q];
        rv = rn, xv = xn;
    }
}

// The same for a constant-density MAC column: six loads a cell instead of
// eight, a plane of them in flight (residuals only, x not written).  B200, from
// 400,000 cells as for FEM: FP32 residual of 192^3 and 96^3 23 -> 15 us, max norm
// 61 -> 41 us at 192^3, FP64 residual to FP32 50 us either way.
template <typename T, typename F>
__device__ __forceinline__ void mac_march(const lvl_dev &L, const T *__restrict__ x, const T *__restrict__ r, int i,
                                          int j, int k0, int k1, F emit) {
    const int sy = L.n0, sz = L.n0 * L.n1;
    const int xl = nb_lo(i, L.n0, L.p0, 1), xh = nb_hi(i, L.n0, L.p0, 1), yl = nb_lo(j, L.n1, L.p1, sy),
              yh = nb_hi(j, L.n1, L.p1, sy);
    const size_t id = i + sy * j + (size_t)sz * k0;
    const T *c = x + id, *q = r + id;
    T zm = c[nb_lo(k0, L.n2, L.p2, sz)], xc = c[0], zp = c[nb_hi(k0, L.n2, L.p2, sz)];
    T xm = c[xl], xp = c[xh], ym = c[yl], yp = c[yh], rv = q[0];
    for (int k = k0; k < k1; k++) {
        T zn = 0, xm1 = 0, xp1 = 0, ym1 = 0, yp1 = 0, rn = 0;
        c += sz, q += sz;
        if (k + 1 < k1) {
            zn = c[nb_hi(k + 1, L.n2, L.p2, sz)];
            xm1 = c[xl], xp1 = c[xh], ym1 = c[yl], yp1 = c[yh], rn = q[0];
        }
        T diag;
        const T s = mac_sum(L, i, j, k, xm, xp, ym, yp, zm, zp, diag);
        emit(k, s, diag, rv, xc);
        zm = xc, xc = zp, zp = zn;
        xm = xm1, xp = xp1, ym = ym1, yp = yp1, rv = rn;
    }
}

// Planes per thread of a phase over `points` points; 1: point by point.  A
// point by itself waits on its 21 loads and little else; marching reads less
// and keeps a plane of loads in flight, but leaves fewer threads.  The line lies
// at 200,000 threads and 16 planes (B200, 193^3 nodes): FP64 residual to FP32
// 126 -> 79 us (8 planes 84, 4 planes 93), its max norm 151 -> 77 us, FP32
// residual of 193^3 and 97^3 38 -> 27 us, FP32 colour pass of 193^3 19 -> 14 us.
// Below it the two are level: FP32 colour pass of 97^3 variable density 5.2 us
// either way, with a quarter of the threads 5.8 us.
inline int march_planes(size_t points) {
    const size_t p = points / 200000;
    return p < 2 ? 1 : p > 16 ? 16 : (int)p;
}

// The Q1 stencil couples a node only to its edge and corner neighbours (the
// face entries are zero), so colouring by the parities of i and j alone never
// puts two coupled nodes in one colour: four colour passes are an exact
// Gauss-Seidel sweep.  The line of a colour has (n0 + 1) / 2 nodes a row for
// either parity of i.
template <typename T, bool MARCH>
__device__ __forceinline__ void body_fem_gs(lvl_dev L, T *x, const T *__restrict__ r, int colour, const T *__restrict__ ri, unsigned inv, int pt, int kb, int pz) {
    const int h = (L.n0 + 1) >> 1, b = line_row(pt, inv);
    const int i = 2 * (pt - b * h) + (colour & 1), j = 2 * b + (colour >> 1);
    if (i >= L.n0 || j >= L.n1) return;
    if (MARCH) {
        const int k0 = kb * pz, k1 = min(k0 + pz, L.n2), h = fem_walls(L, i, j);
        const int id0 = i + L.n0 * j, sz = L.n0 * L.n1;
        if (ri)
            fem_march<T, true, false>(L, x, r, ri, i, j, k0, k1,
                                      [&](int k, T s, T diag, T rv, T) { x[id0 + sz * k] = (rv - s) / diag; });
        else
            fem_march<T, false, false>(L, x, r, ri, i, j, k0, k1, [&](int k, T s, T, T rv, T) {
                const int w = h + (!L.p2 && (k == 0 || k == L.n2 - 1) ? 1 : 0);
                x[id0 + sz * k] = (rv - s) * ((T)(1 << w) * (T)0.03125);
            });
        return;
    }
    const int k = kb;
    T diag;
    const int id = i + L.n0 * (j + L.n1 * k);
    if (ri) {
        const T s = fem_offdiag_vd(L, x, ri, i, j, k, diag);
        x[id] = (r[id] - s) / diag;
    } else {
        const T s = fem_offdiag(L, x, i, j, k, diag);
        x[id] = (r[id] - s) * fem_inv_diag<T>(L, i, j, k);
    }
}

// ---- residuals: r - A x into emit(index, value) ------------------------------
template <typename T, int KIND, bool MARCH, typename F>
__device__ __forceinline__ void body_resid_emit(const lvl_dev &L, const T *__restrict__ x, const T *__restrict__ r,
                                                const T *__restrict__ ri, unsigned inv, int pt, int kb, int pz, F emit) {
    const int j = line_row(pt, inv), i = pt - j * L.n0;
    if (j >= L.n1) return;
    if (MARCH) {  // MAC: constant density
        const int k0 = kb * pz, k1 = min(k0 + pz, L.n2), id0 = i + L.n0 * j, sz = L.n0 * L.n1;
        auto f = [&](int k, T s, T diag, T rv, T xv) { emit(id0 + sz * k, rv - s - diag * xv); };
        if (KIND == 0) mac_march<T>(L, x, r, i, j, k0, k1, f);
        else if (ri) fem_march<T, true, true>(L, x, r, ri, i, j, k0, k1, f);
        else fem_march<T, false, true>(L, x, r, ri, i, j, k0, k1, f);
        return;
    }
    const int k = kb;
    T diag;
    const T s = op_offdiag<T>(KIND, L, x, ri, i, j, k, diag);
    const int id = i + L.n0 * (j + L.n1 * k);
    emit(id, r[id] - s - diag * x[id]);
}

// res = r - A x
template <typename T, int KIND, bool MARCH>
__device__ __forceinline__ void body_resid(lvl_dev L, const T *__restrict__ x, const T *__restrict__ r,
                                           T *__restrict__ res, const T *__restrict__ ri, unsigned inv, int pt, int k, int pz) {
    body_resid_emit<T, KIND, MARCH>(L, x, r, ri, inv, pt, k, pz, [&](int id, T v) { res[id] = v; });
}

// max |r - A x| over the calling thread's points, as the ordered bit pattern
// (NaN the largest)
template <int KIND, bool MARCH>
__device__ __forceinline__ unsigned long long body_resid_max(lvl_dev L, const double *__restrict__ x,
                                                             const double *__restrict__ r,
                                                             const double *__restrict__ ri, unsigned inv, int pt,
                                                             int k, int pz) {
    unsigned long long m = 0;
    body_resid_emit<double, KIND, MARCH>(L, x, r, ri, inv, pt, k, pz, [&](int, double v) {
        const double a = fabs(v);
        const unsigned long long b = a != a ? 0x7ff8000000000000ULL : (unsigned long long)__double_as_longlong(a);
        m = b > m ? b : m;
    });
    return m;
}

// The mixed form's FP64 residual handed to the FP32 cycle in one pass: the
// residual r - A x in FP64, rounded to FP32 as the cycle's right-hand side,
// and the cycle's FP32 start value zeroed.
template <int KIND, bool MARCH>
__device__ __forceinline__ void body_resid_to_f32(lvl_dev L, const double *__restrict__ x,
                                                  const double *__restrict__ r, const double *__restrict__ ri,
                                                  float *__restrict__ rs, float *__restrict__ xs, unsigned inv,
                                                  int pt, int k, int pz) {
    body_resid_emit<double, KIND, MARCH>(L, x, r, ri, inv, pt, k, pz, [&](int id, double v) {
        rs[id] = (float)v;
        xs[id] = 0;
    });
}

// the block's maximum of b into *mx: one atomic per block, none where the
// maximum so far already covers it.  Every thread of the block calls it.  B200,
// 192^3, by ncu: the right-hand side's norm 16 us, with an atomic per warp 19;
// the marching residual norms take 41 (MAC) and 75 us (FEM) either way.
__device__ __forceinline__ void block_max_into(unsigned long long b, unsigned long long *mx) {
    __shared__ unsigned long long wmax[32];
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
        b = t > b ? t : b;
    }
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nw = (blockDim.x * blockDim.y * blockDim.z) >> 5;
    if ((tid & 31) == 0) wmax[tid >> 5] = b;
    __syncthreads();
    if (tid < 32) {
        b = tid < nw ? wmax[tid] : 0;
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o);
            b = t > b ? t : b;
        }
        if (tid == 0 && b > *(volatile unsigned long long *)mx) atomicMax(mx, b);
    }
}

// max |r| over a grid-stride range, as the ordered bit pattern (NaN the largest)
__device__ __forceinline__ unsigned long long body_absmax(const double *__restrict__ r, size_t n, size_t t0, size_t ts) {
    unsigned long long m = 0;
#pragma unroll 4
    for (size_t i = t0; i < n; i += ts) {
        const double a = fabs(r[i]);
        const unsigned long long b = a != a ? 0x7ff8000000000000ULL : (unsigned long long)__double_as_longlong(a);
        m = b > m ? b : m;
    }
    return m;
}

// ---- grid transfer ---------------------------------------------------------
template <typename T>
__device__ __forceinline__ void body_mac_restrict(lvl_dev F, lvl_dev C, const T *__restrict__ res, T *__restrict__ rc,
                               T *__restrict__ xc0, int bx_, int by_, int bz_) {
    int I = bx_ * blockDim.x + threadIdx.x;
    int J = by_ * blockDim.y + threadIdx.y;
    int K = bz_ * blockDim.z + threadIdx.z;
    if (I >= C.n0 || J >= C.n1 || K >= C.n2) return;
    T s = 0;
    for (int c = 0; c < 2; c++)
        for (int b = 0; b < 2; b++)
            for (int a = 0; a < 2; a++) s += res[(2 * I + a) + F.n0 * ((2 * J + b) + F.n1 * (2 * K + c))];
    rc[I + C.n0 * (J + C.n1 * K)] = (T)0.5 * s;
    xc0[I + C.n0 * (J + C.n1 * K)] = 0;
}

// x += the interpolated coarse correction.  A thread takes the 2 x 2 fine
// points (j, k) around one pair of coarse rows at its i: they share their
// coarse values (18 loads for four points instead of 32; FEM 8 instead of up
// to 27), and each point's sum keeps its order.  FEM, 193^3 and 97^3 levels:
// 101 -> 15 us a launch; its DRAM floor is 9 us.
template <typename T>
__device__ __forceinline__ void body_mac_prolong(lvl_dev F, lvl_dev C, T *__restrict__ x, const T *__restrict__ xc, int bx_, int by_, int bz_) {
    const int i = bx_ * blockDim.x + threadIdx.x;
    const int J = by_ * blockDim.y + threadIdx.y;
    const int K = bz_ * blockDim.z + threadIdx.z;
    if (i >= F.n0 || J >= C.n1 || K >= C.n2) return;
    const int I = i >> 1, In = wrapi(I + ((i & 1) ? 1 : -1), C.n0, C.p0);
    const T wx[2] = {In < 0 ? (T)1 : (T)0.75, In < 0 ? (T)0 : (T)0.25};
    const int ix = In < 0 ? I : In;
    int jy[3], kz[3];
    bool oy[3], oz[3];
#pragma unroll
    for (int o = 0; o < 3; o++) {
        const int a = wrapi(J + o - 1, C.n1, C.p1), b = wrapi(K + o - 1, C.n2, C.p2);
        oy[o] = a >= 0;
        oz[o] = b >= 0;
        jy[o] = a < 0 ? J : a;
        kz[o] = b < 0 ? K : b;
    }
    T v[3][3][2];
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int b = 0; b < 3; b++) {
            const T *row = xc + (size_t)C.n0 * (jy[b] + (size_t)C.n1 * kz[c]);
            v[c][b][0] = row[I];
            v[c][b][1] = row[ix];
        }
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int k = 2 * K + c;
        if (k >= F.n2) continue;
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int j = 2 * J + b;
            if (j >= F.n1) continue;
            // odd points lean on the next coarse cell, even ones on the
            // previous; without it the near cell counts fully
            const int nb = b ? 2 : 0, nc = c ? 2 : 0;
            const T wy[2] = {oy[nb] ? (T)0.75 : (T)1, oy[nb] ? (T)0.25 : (T)0};
            const T wz[2] = {oz[nc] ? (T)0.75 : (T)1, oz[nc] ? (T)0.25 : (T)0};
            T e = 0;
#pragma unroll
            for (int q = 0; q < 8; q++) {
                const int qa = q & 1, qb = (q >> 1) & 1, qc = q >> 2;
                const T wt = wx[qa] * wy[qb] * wz[qc];
                if (wt != 0) e += wt * v[qc ? nc : 1][qb ? nb : 1][qa];
            }
            x[i + F.n0 * (j + F.n1 * k)] += e;
        }
    }
}

template <typename T>
__device__ __forceinline__ void body_fem_restrict(lvl_dev F, lvl_dev C, const T *__restrict__ res, T *__restrict__ rc,
                               T *__restrict__ xc0, int bx_, int by_, int bz_) {
    int I = bx_ * blockDim.x + threadIdx.x;
    int J = by_ * blockDim.y + threadIdx.y;
    int K = bz_ * blockDim.z + threadIdx.z;
    if (I >= C.n0 || J >= C.n1 || K >= C.n2) return;
    const int nf[3] = {F.n0, F.n1, F.n2}, p[3] = {F.p0, F.p1, F.p2};
    const int c[3] = {I, J, K};
    int idx[3][3];
    T w[3][3];
    for (int d = 0; d < 3; d++)
        for (int o = -1; o <= 1; o++) {
            int v = wrapi(2 * c[d] + o, nf[d], p[d]);
            idx[d][o + 1] = v;
            w[d][o + 1] = (v < 0) ? (T)0 : (o == 0 ? (T)1 : (T)0.5);
        }
    T s = 0;
    for (int oc = 0; oc < 3; oc++) {
        if (idx[2][oc] < 0) continue;
        for (int ob = 0; ob < 3; ob++) {
            if (idx[1][ob] < 0) continue;
            for (int oa = 0; oa < 3; oa++) {
                if (idx[0][oa] < 0) continue;
                s += w[0][oa] * w[1][ob] * w[2][oc] * res[idx[0][oa] + F.n0 * (idx[1][ob] + F.n1 * idx[2][oc])];
            }
        }
    }
    rc[I + C.n0 * (J + C.n1 * K)] = (T)0.5 * s;
    xc0[I + C.n0 * (J + C.n1 * K)] = 0;
}

template <typename T>
__device__ __forceinline__ void body_fem_prolong(lvl_dev F, lvl_dev C, T *__restrict__ x, const T *__restrict__ xc, int bx_, int by_, int bz_) {
    const int i = bx_ * blockDim.x + threadIdx.x;
    const int J = by_ * blockDim.y + threadIdx.y;
    const int K = bz_ * blockDim.z + threadIdx.z;
    if (i >= F.n0 || J >= C.n1 || K >= C.n2) return;
    const bool odd = i & 1;
    const int I = i >> 1, I1 = odd ? wrapi(I + 1, C.n0, C.p0) : I;
    // beyond a wall there is no point that would use the next row or plane
    const int J1 = max(wrapi(J + 1, C.n1, C.p1), 0), K1 = max(wrapi(K + 1, C.n2, C.p2), 0);
    const T wx = odd ? (T)0.5 : (T)1;
    T v[2][2][2];
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const T *row = xc + (size_t)C.n0 * ((b ? J1 : J) + (size_t)C.n1 * (c ? K1 : K));
            v[c][b][0] = row[I];
            v[c][b][1] = row[I1];
        }
#pragma unroll
    for (int c = 0; c < 2; c++) {
        const int k = 2 * K + c;
        if (k >= F.n2) continue;
#pragma unroll
        for (int b = 0; b < 2; b++) {
            const int j = 2 * J + b;
            if (j >= F.n1) continue;
            const T w = wx * (b ? (T)0.5 : (T)1) * (c ? (T)0.5 : (T)1);
            T e = 0;
#pragma unroll
            for (int qc = 0; qc <= c; qc++)
#pragma unroll
                for (int qb = 0; qb <= b; qb++) {
                    e += w * v[qc][qb][0];
                    if (odd) e += w * v[qc][qb][1];
                }
            x[i + F.n0 * (j + F.n1 * k)] += e;
        }
    }
}

// coarsest grid: x = B r with the precomputed dense inverse B (row-major)
template <typename T>
__device__ __forceinline__ void body_coarse_dense(int np, const double *__restrict__ B, T *__restrict__ x,
                                                  const T *__restrict__ r, int bx_, int gx_) {
    __shared__ double rs[1024];
    for (int p = threadIdx.x; p < np; p += blockDim.x) rs[p] = (double)r[p];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int row = bx_ * (blockDim.x >> 5) + warp; row < np; row += gx_ * (blockDim.x >> 5)) {
        const double *b = B + (size_t)row * np;
        double acc = 0;
        for (int c = lane; c < np; c += 32) acc += b[c] * rs[c];
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) x[row] = (T)acc;
    }
}

// coarsest grid fallback: many Gauss-Seidel sweeps inside one thread block
template <typename T, int KIND>
__device__ __forceinline__ void body_coarse_solve(lvl_dev L, T *__restrict__ x, const T *__restrict__ r, int sweeps) {
    const int np = L.n0 * L.n1 * L.n2;
    for (int p = threadIdx.x; p < np; p += blockDim.x) x[p] = 0;
    __syncthreads();
    const int ncol = (KIND == 0) ? 2 : 8;
    for (int s = 0; s < sweeps; s++)
        for (int col = 0; col < ncol; col++) {
            for (int p = threadIdx.x; p < np; p += blockDim.x) {
                int i = p % L.n0, j = (p / L.n0) % L.n1, k = p / (L.n0 * L.n1);
                int my = (KIND == 0) ? ((i + j + k) & 1) : ((i & 1) | ((j & 1) << 1) | ((k & 1) << 2));
                if (my != col) continue;
                T diag;
                T sum = (KIND == 0) ? mac_offdiag(L, x, i, j, k, diag) : fem_offdiag(L, x, i, j, k, diag);
                x[p] = (r[p] - sum) / diag;
            }
            __syncthreads();
        }
}

// FP64 <-> FP32 helpers of the mixed form
__device__ __forceinline__ void body_to_f32(const double *__restrict__ a, float *__restrict__ b, size_t n, int bx_) {
    size_t i = bx_ * (size_t)blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}
// two elements a thread (the level arrays start on 256-byte boundaries)
__device__ __forceinline__ void body_add_f32(double *__restrict__ a, const float *__restrict__ b, size_t n, int bx_) {
    const size_t i = 2 * (bx_ * (size_t)blockDim.x + threadIdx.x);
    if (i + 1 < n) {
        double2 v = *reinterpret_cast<double2 *>(a + i);
        const float2 w = *reinterpret_cast<const float2 *>(b + i);
        v.x += (double)w.x;
        v.y += (double)w.y;
        *reinterpret_cast<double2 *>(a + i) = v;
    } else if (i < n) {
        a[i] += (double)b[i];
    }
}
template <typename T>
__device__ __forceinline__ void body_zero(T *a, size_t n, int bx_) {
    size_t i = bx_ * (size_t)blockDim.x + threadIdx.x;
    if (i < n) a[i] = 0;
}


// ---- the control of one solve (mg_prob::run, Utilities/mg_probs.cc:3-83) ---
__device__ __forceinline__ void mg_begin_state(mg_ctl *c, unsigned long long *mx) {
    c->phase = 0;
    c->todo = c->iV / kMgIP;
    if (c->todo < 1) c->todo = 1;
    c->extra = 0;
    c->it = 0;
    c->count = 0;
    c->gave_up = 0;
    c->active = 1;
    c->need_res = c->todo == 1;
    mx[0] = 0;
    mx[1] = 0;
}

// One step of the control after an iteration, with the fine-level max-norm
// residual in mx[0] (and max |rhs| in mx[1] for the relative tolerance);
// returns true when the solve is finished (the predictor is then updated).
__device__ __forceinline__ bool mg_ctl_step(mg_ctl *c, unsigned long long *mx, double tol, double rtol, int exact) {
    const double r = __longlong_as_double((long long)mx[0]);
    mx[0] = 0;
    // the mixed form's relative tolerance (mixed_rtol x max |rhs|)
    const double rhs = __longlong_as_double((long long)mx[1]);
    const double tol_eff = (rtol > 0 && rtol * rhs > tol) ? rtol * rhs : tol;
    c->count++;
    c->cycles_total++;
    bool done = false;
    if (c->phase <= 1) {
        if (--c->todo <= 0) {
            c->res_out = r;
            if (r > tol_eff && c->extra < 20) {
                c->extra++;
                c->todo = c->extra;
                c->phase = 1;
            } else if (rtol > 0 && !exact) {
                done = true;  // the relaxed form skips the insurance cycles
            } else {
                c->phase = 2;
                c->todo = 2;
            }
        }
    } else if (c->phase == 2) {
        if (--c->todo <= 0) {
            if (exact) {
                c->prev = 1e300;
                c->res_out = r;
                c->it = 0;
                if (r > 0 && r < 0.7 * c->prev) c->phase = 3;
                else done = true;
            } else {
                done = true;
            }
        }
    } else {
        c->prev = c->res_out;
        c->res_out = r;
        c->it++;
        if (!(c->it < 60 && r > 0 && r < 0.7 * c->prev)) done = true;
    }
    if (c->count >= kMgMaxCycles) done = true;
    if (done) {
        // mg_pred::update (alpha = 0)
        const double alpha = 1 / (3 * kMgIP);
        double dV = c->iV - c->V_avg;
        int exreduce = static_cast<int>(dV / sqrt(c->V_var));
        exreduce = exreduce > 0 ? exreduce : 0;
        c->iV += kMgIP * c->extra * (c->extra + 1) / 2 - 1 - exreduce;
        if (c->iV < kMgIP) c->iV = 2 * kMgIP - 1;
        c->V_avg = (1 - alpha) * c->V_avg + alpha * c->iV;
        c->V_var = (1 - alpha) * (c->V_var + alpha * dV * dV);
        c->last_cycles = c->count;
        c->active = 0;
        c->nan = c->res_out != c->res_out || c->gave_up;
    }
    // the residual is read only where a phase ends (and every cycle of the
    // stagnation loop): the next iteration computes it only then
    c->need_res = (c->phase <= 1 && c->todo == 1) || (c->phase == 2 && c->todo == 1 && exact) || c->phase == 3;
    return done;
}

}  // namespace rmt3d
