// FEM colour passes and residuals, and MAC residuals, that march along z
// (fem_march and mac_march, mg_body.cuh) against the same phases point by point: the same bits for every mix of
// periodic and walled axes, both densities, both types and every number of
// planes a thread, the last block short.  Built with the address sanitizer,
// each array a heap block of its own size.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include <cuda_runtime.h>

struct dim {
    int x, y, z;
};
static dim threadIdx{0, 0, 0}, blockDim{1, 1, 1};
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }
inline long long __double_as_longlong(double v) {
    long long b;
    memcpy(&b, &v, 8);
    return b;
}
inline double __longlong_as_double(long long b) {
    double v;
    memcpy(&v, &b, 8);
    return v;
}
template <typename V>
V __shfl_xor_sync(unsigned, V v, int) {
    return v;
}
inline void __syncthreads() {}
inline unsigned long long atomicMax(unsigned long long *p, unsigned long long v) {
    const unsigned long long o = *p;
    if (v > o) *p = v;
    return o;
}
template <typename V>
V min(V a, V b) {
    return a < b ? a : b;
}
template <typename V>
V max(V a, V b) {
    return a > b ? a : b;
}

#include "mg_body.cuh"

using namespace rmt3d;

template <typename T>
static bool same(const std::vector<T> &a, const std::vector<T> &b) {
    return memcmp(a.data(), b.data(), a.size() * sizeof(T)) == 0;
}

// blocks of 256 threads over a line of `line` points, pz planes a thread
template <typename F>
static void run(int line, int n2, int pz, F f) {
    for (int kb = 0; kb < (n2 + pz - 1) / pz; kb++)
        for (int pt = 0; pt < (line + 255) / 256 * 256; pt++) f(pt, kb);
}

template <typename T>
static int check(const int *n, int axes, bool vd) {
    const lvl_dev L{n[0], n[1], n[2], axes & 1, (axes >> 1) & 1, (axes >> 2) & 1};
    const size_t N = (size_t)n[0] * n[1] * n[2];
    const size_t nc = (size_t)(n[0] - !L.p0) * (n[1] - !L.p1) * (n[2] - !L.p2);
    std::mt19937 gen(axes + 8 * vd + n[0]);
    std::uniform_real_distribution<double> U(-1, 1);
    std::vector<T> x(N), r(N), ri(nc);
    for (T &v : x) v = (T)U(gen);
    for (T &v : r) v = (T)U(gen);
    for (T &v : ri) v = (T)(1.2 + U(gen));
    const T *q = vd ? ri.data() : nullptr;
    const int h = (n[0] + 1) / 2, rows = (n[1] + 1) / 2;
    std::vector<T> want(x), res(N);
    for (int c = 0; c < 4; c++)
        run(h * rows, n[2], 1, [&](int pt, int kb) {
            body_fem_gs<T, false>(L, want.data(), r.data(), c, q, line_inv(h), pt, kb, 1);
        });
    run(n[0] * n[1], n[2], 1, [&](int pt, int kb) {
        body_resid<T, 1, false>(L, x.data(), r.data(), res.data(), q, line_inv(n[0]), pt, kb, 1);
    });
    // constant-density MAC residual (any box of at least two cells an axis)
    std::vector<T> mres(N);
    run(n[0] * n[1], n[2], 1, [&](int pt, int kb) {
        body_resid<T, 0, false>(L, x.data(), r.data(), mres.data(), nullptr, line_inv(n[0]), pt, kb, 1);
    });
    for (int pz = 1; pz <= 16; pz++) {
        std::vector<T> gm(N);
        run(n[0] * n[1], n[2], pz, [&](int pt, int kb) {
            body_resid<T, 0, true>(L, x.data(), r.data(), gm.data(), nullptr, line_inv(n[0]), pt, kb, pz);
        });
        if (!same(gm, mres)) {
            printf("%d %d %d axes %d planes %d: MAC residual\n", n[0], n[1], n[2], axes, pz);
            return 1;
        }
    }
    for (int pz = 1; pz <= 16; pz++) {
        std::vector<T> got(x), gres(N);
        for (int c = 0; c < 4; c++)
            run(h * rows, n[2], pz, [&](int pt, int kb) {
                body_fem_gs<T, true>(L, got.data(), r.data(), c, q, line_inv(h), pt, kb, pz);
            });
        run(n[0] * n[1], n[2], pz, [&](int pt, int kb) {
            body_resid<T, 1, true>(L, x.data(), r.data(), gres.data(), q, line_inv(n[0]), pt, kb, pz);
        });
        if (!same(got, want) || !same(gres, res)) {
            printf("%d %d %d axes %d vd %d planes %d: %s\n", n[0], n[1], n[2], axes, vd, pz,
                   same(got, want) ? "residual" : "colour passes");
            return 1;
        }
    }
    return 0;
}

int main() {
    // nodes per axis: odd with walls, even where periodic
    const int sizes[][3] = {{3, 5, 3}, {9, 7, 17}, {5, 33, 11}};
    int bad = 0;
    for (auto &s : sizes)
        for (int axes = 0; axes < 8; axes++) {
            int n[3];
            for (int d = 0; d < 3; d++) n[d] = s[d] - ((axes >> d) & 1);
            for (int vd = 0; vd < 2; vd++) bad += check<double>(n, axes, vd) + check<float>(n, axes, vd);
        }
    return bad != 0;
}
