// Runs the device code of the shared-memory V-cycle (mg_slab.cuh) on host
// threads -- one per CUDA thread, a cluster of small CTAs -- and compares it
// bit for bit with the per-phase V-cycle of mg_ops.cuh, and that operator with
// its term-by-term form (ref_ops.inc).  Built with the
// address sanitizer, every CTA's shared memory a heap block of its own size,
// so an index outside it ends the run.
//   slab_sim kind(0 MAC, 1 FEM) vd f64 n0 n1 n2 p0 p1 p2 csize v_down v_up l0 seed [drop]
// With `drop`, that value of those sent to CTA 1 is lost, so its wait gives
// up: every thread still ends, no mbarrier is armed twice in a phase, CTA 1's planes
// come out NaN and the solve's control, given that residual, reports NaN.
#include <atomic>
#include <barrier>
#include <chrono>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <thread>

#include <cuda_runtime.h>

#define RMT3D_SLAB_THREADS 32
namespace {
struct cta_state {
    unsigned char *smem = nullptr;
    size_t bytes = 0;
    double lane[32];
    std::barrier<> *bar = nullptr;
};
std::vector<cta_state> g_cta;
std::barrier<> *g_all = nullptr;
thread_local int t_rank = 0;
struct dim {
    int x, y, z;
};
}  // namespace
thread_local dim threadIdx{0, 0, 0}, blockDim{1, 1, 1};
inline void __syncthreads() {
    if (!g_cta.empty()) g_cta[t_rank].bar->arrive_and_wait();
}
inline double __shfl_xor_sync(unsigned, double v, int o) {
    if (g_cta.empty()) return v;  // the one-thread reference run
    cta_state &c = g_cta[t_rank];
    c.lane[threadIdx.x] = v;
    c.bar->arrive_and_wait();
    const double r = c.lane[threadIdx.x ^ o];
    c.bar->arrive_and_wait();
    return r;
}
// for the control (mg_body.cuh)
inline unsigned long long __shfl_xor_sync(unsigned, unsigned long long v, int) { return v; }
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
inline unsigned long long atomicMax(unsigned long long *p, unsigned long long v) {
    const unsigned long long o = *p;
    if (v > o) *p = v;
    return o;
}
inline unsigned __umulhi(unsigned a, unsigned b) { return (unsigned)(((uint64_t)a * b) >> 32); }

// the cluster primitives on host threads (in place of cluster_ops.cuh)
#include <vector>
namespace rmt3d {
inline void cl_barrier() { g_all->arrive_and_wait(); }
inline unsigned cl_rank() { return (unsigned)t_rank; }
template <typename T>
T *cl_map(T *p, unsigned rank) {
    if (rank >= g_cta.size()) abort();
    return (T *)(g_cta[rank].smem + ((unsigned char *)p - g_cta[t_rank].smem));
}
typedef uintptr_t cl_addr;
template <typename T>
cl_addr cl_remote(T *p, unsigned rank) {
    return (cl_addr)cl_map(p, rank);
}
// an mbarrier as {bytes still expected, completed phases}; an unarmed phase
// holds kUnarmed more, so that early sends cannot complete it
struct sim_bar {
    std::atomic<int> due, phase;
};
constexpr int kUnarmed = 1 << 28;
inline void sim_step(sim_bar *b, int d) {
    if (b->due.fetch_add(d) + d == 0) {
        b->due.fetch_add(kUnarmed);
        b->phase.fetch_add(1);
    }
}
int g_drop = -1;  // which value sent to CTA 1 is lost (-1: none)
std::atomic<int> g_sent{0}, g_rearmed{0};
template <typename T>
void cl_send(cl_addr a, T v, cl_addr bar) {
    const bool to1 = g_drop >= 0 && (unsigned char *)bar >= g_cta[1].smem && (unsigned char *)bar < g_cta[1].smem + g_cta[1].bytes;
    if (to1 && g_sent.fetch_add(1) == g_drop) return;
    *(T *)a = v;
    sim_step((sim_bar *)bar, -(int)sizeof(T));
}
inline void halo_init(uint64_t *b) {
    ((sim_bar *)b)->due = kUnarmed;
    ((sim_bar *)b)->phase = 0;
}
inline void halo_init_fence() {}
inline void halo_arm(uint64_t *b, unsigned bytes) {
    if (((sim_bar *)b)->due < kUnarmed / 2) g_rearmed++;  // the phase's one arrival has come already
    sim_step((sim_bar *)b, (int)bytes - kUnarmed);
}
inline bool halo_wait(uint64_t *b, unsigned parity) {
    for (int it = 0; it < (g_drop < 0 ? 4000000 : 8000); it++) {
        if ((((sim_bar *)b)->phase & 1) != (int)parity) return true;
        std::this_thread::sleep_for(std::chrono::microseconds(20));
    }
    return false;
}
inline void cl_linger() {}
int fail(int code, const std::string &) { return code; }
}  // namespace rmt3d
#include "mg_slab.cuh"

using std::max;
using std::min;
#include "mg_body.cuh"

namespace rmt3d {
#include "ref_ops.inc"
}
using namespace rmt3d;

// one row of the operator, as the kernels form it and term by term: the same
// updated value and residual
template <typename T, int KIND, bool VD>
static size_t check_rows(const pmg_level &P, T rv) {
    const lvl_dev L = ldev(P);
    const T *x = LX<T>(P), *ri = VD ? LRI<T>(P) : nullptr;
    size_t bad = 0;
    for (int k = 0; k < L.n2; k++)
        for (int j = 0; j < L.n1; j++)
            for (int i = 0; i < L.n0; i++) {
                T d1, d2;
                const T s1 = op_offdiag<T>(KIND, L, x, ri, i, j, k, d1);
                const T s2 = KIND ? (VD ? ref_fem_offdiag_vd(L, x, ri, i, j, k, d2) : ref_fem_offdiag(L, x, i, j, k, d2))
                                  : (VD ? ref_mac_offdiag_vd(L, x, ri, i, j, k, d2) : ref_mac_offdiag(L, x, i, j, k, d2));
                const T a = (rv - s1) / d1, b = (rv - s2) / d2;
                if (memcmp(&a, &b, sizeof(T)) || memcmp(&d1, &d2, sizeof(T)) || s1 != s2) bad++;
            }
    return bad;
}

static int plan(int kind, const int n[3], const int prd[3], std::vector<mg_level> &lv) {
    mg_level L;
    for (int d = 0; d < 3; d++) L.n[d] = n[d], L.prd[d] = prd[d];
    lv.push_back(L);
    while (lv.back().npts() > (size_t)kDensePts) {
        mg_level c;
        bool ok = true;
        for (int d = 0; d < 3; d++) {
            const int len = lv.back().n[d];
            c.prd[d] = prd[d];
            if (kind == 0 || prd[d]) {
                ok = ok && len % 2 == 0 && len >= 4;
                c.n[d] = len / 2;
            } else {
                ok = ok && len % 2 == 1 && len >= 3;
                c.n[d] = (len - 1) / 2 + 1;
            }
        }
        if (!ok) break;
        lv.push_back(c);
    }
    return lv.back().npts() <= (size_t)kDenseMax ? 0 : 1;
}

template <typename T, int KIND, bool VD>
static int run(const std::vector<mg_level> &lv, int csize, int vdn, int vup, int l0, unsigned seed, bool load_x) {
    std::mt19937_64 rng(seed);
    std::uniform_real_distribution<double> U(-1, 1);
    pmg_args A;
    memset(&A, 0, sizeof(A));
    A.kind = KIND;
    A.nlev = (int)lv.size();
    A.v_down = vdn;
    A.v_up = vup;
    std::vector<std::vector<T>> x, r, s, ri;
    for (auto &l : lv) {
        x.emplace_back(l.npts(), (T)0), r.emplace_back(l.npts(), (T)0), s.emplace_back(l.npts(), (T)0);
        ri.emplace_back(l.npts(), (T)0);
        for (auto &v : ri.back()) v = (T)(1.0 + 0.2 * U(rng));
    }
    for (auto &v : r[l0]) v = (T)U(rng);
    if (load_x)
        for (auto &v : x[l0]) v = (T)U(rng);
    const size_t np = lv.back().npts();
    std::vector<double> B(np * np);
    for (auto &v : B) v = U(rng) / np;
    A.dense = B.data();
    int gave_up = 0;
    A.gave_up = &gave_up;
    for (int l = 0; l < A.nlev; l++) {
        for (int d = 0; d < 3; d++) A.lv[l].n[d] = lv[l].n[d], A.lv[l].prd[d] = lv[l].prd[d];
        set_level_ptrs<T>(A.lv[l], x[l].data(), r[l].data(), s[l].data());
        if (VD) (sizeof(T) == 8 ? (void)(A.lv[l].ri = (double *)ri[l].data()) : (void)(A.lv[l].ris = (float *)ri[l].data()));
    }
    for (int l = 0; l < A.nlev; l++) {
        const std::vector<T> keep_x = x[l];
        for (auto &v : x[l]) v = (T)U(rng);
        if (size_t bad = check_rows<T, KIND, VD>(A.lv[l], (T)0.37)) {
            printf("level %d: %zu rows differ from the term-by-term operator\n", l, bad);
            return 5;
        }
        x[l] = keep_x;
    }
    const std::vector<T> x0 = x[l0];
    slab_args S;
    const size_t bytes = slab_layout(lv, l0, csize, sizeof(T) == 8, VD, load_x, &S);
    if (!bytes) return 2;
    g_cta.assign(csize, cta_state());
    for (auto &c : g_cta) {
        c.smem = (unsigned char *)aligned_alloc(16, (bytes + 15) & ~(size_t)15);
        c.bytes = bytes;
        memset(c.smem, 0xff, bytes);  // NaN: reads of what was never written show
        c.bar = new std::barrier<>(RMT3D_SLAB_THREADS);
    }
    g_all = new std::barrier<>(csize * RMT3D_SLAB_THREADS);
    std::vector<std::thread> th;
    for (int b = 0; b < csize; b++)
        for (int t = 0; t < RMT3D_SLAB_THREADS; t++)
            th.emplace_back([&, b, t]() {
                t_rank = b;
                threadIdx.x = t;
                slab_cycle<T, KIND, VD>(A, S, g_cta[b].smem);
            });
    for (auto &t : th) t.join();
    const std::vector<T> got = x[l0];
    for (auto &c : g_cta) {
        free(c.smem);
        delete c.bar;
    }
    g_cta.clear();
    if (g_drop >= 0) {
        const slab_level &L = S.lv[0];
        const size_t pl = (size_t)L.n0 * L.n1;
        size_t numbers = 0;
        for (size_t q = pl * L.q; q < pl * std::min(2 * L.q, L.n2); q++) numbers += got[q] == got[q];
        // the control at the end of the solve (its last cycles read no residual)
        mg_ctl c;
        memset(&c, 0, sizeof(c));
        unsigned long long mx[2] = {0, 0};
        mg_begin_state(&c, mx);
        c.phase = 2;
        c.todo = 1;
        c.gave_up = gave_up;
        const bool done = mg_ctl_step(&c, mx, 1, 0, 0);
        printf("given up %d, armed twice %d, numbers in CTA 1's planes %zu, nan %d\n", gave_up, g_rearmed.load(), numbers, c.nan);
        return gave_up && !g_rearmed && !numbers && done && c.nan ? 0 : 6;
    }
    x[l0] = x0;
    // the per-phase cycle, one thread; the dense solve in 32 lanes' order
    threadIdx.x = 0;
    blockDim.x = 1;
    const int nc = KIND == 0 ? 2 : 4;
    for (int l = l0; l < A.nlev - 1; l++) {
        const pmg_level &F = A.lv[l], &C = A.lv[l + 1];
        for (int q = 0; q < vdn * nc; q++)
            ph_smooth_colour<T>(KIND, ldev(F), LX<T>(F), LR<T>(F), LRI<T>(F), q % nc, 0, 1);
        ph_resid<T>(KIND, ldev(F), LX<T>(F), LR<T>(F), LS<T>(F), LRI<T>(F), 0, 1);
        ph_restrict<T>(KIND, ldev(F), ldev(C), LS<T>(F), LR<T>(C), LX<T>(C), 0, 1);
    }
    for (size_t row = 0; row < np; row++) {
        double acc[32] = {0};
        for (int lane = 0; lane < 32; lane++)
            for (size_t c = lane; c < np; c += 32) acc[lane] += B[row * np + c] * (double)r[A.nlev - 1][c];
        for (int o = 16; o > 0; o >>= 1) {
            double t[32];
            for (int lane = 0; lane < 32; lane++) t[lane] = acc[lane] + acc[lane ^ o];
            memcpy(acc, t, sizeof(t));
        }
        x[A.nlev - 1][row] = (T)acc[0];
    }
    for (int l = A.nlev - 2; l >= l0; l--) {
        const pmg_level &F = A.lv[l], &C = A.lv[l + 1];
        ph_prolong<T>(KIND, ldev(F), ldev(C), LX<T>(F), LX<T>(C), 0, 1);
        for (int q = 0; q < vup * nc; q++)
            ph_smooth_colour<T>(KIND, ldev(F), LX<T>(F), LR<T>(F), LRI<T>(F), q % nc, 0, 1);
    }
    size_t bad = 0;
    for (size_t q = 0; q < got.size(); q++)
        if (memcmp(&got[q], &x[l0][q], sizeof(T))) {
            if (!bad) printf("first difference at %zu: %.17g %.17g\n", q, (double)got[q], (double)x[l0][q]);
            bad++;
        }
    if (gave_up || g_rearmed) return 7;
    printf("levels %d points %zu bytes/CTA %zu different %zu\n", A.nlev - l0, got.size(), bytes, bad);
    return bad ? 1 : 0;
}

int main(int argc, char **argv) {
    if (argc != 15 && argc != 16) return 3;
    int a[14];
    for (int i = 0; i < 14; i++) a[i] = atoi(argv[i + 1]);
    if (argc == 16) g_drop = atoi(argv[15]);
    const int n[3] = {a[3], a[4], a[5]}, prd[3] = {a[6], a[7], a[8]};
    std::vector<mg_level> lv;
    if (plan(a[0], n, prd, lv)) return 4;
    const bool load = a[12] == 0 && a[2];
#define GO(T, K, V) return run<T, K, V>(lv, a[9], a[10], a[11], a[12], (unsigned)a[13], load)
    if (a[2]) {
        if (a[0]) { if (a[1]) GO(double, 1, true); GO(double, 1, false); }
        if (a[1]) GO(double, 0, true);
        GO(double, 0, false);
    }
    if (a[0]) { if (a[1]) GO(float, 1, true); GO(float, 1, false); }
    if (a[1]) GO(float, 0, true);
    GO(float, 0, false);
}
