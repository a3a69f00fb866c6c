// Kernels and launches of the shared-memory part of a V-cycle (mg_slab.cuh).
#include <algorithm>
#include <mutex>

#include "host_common.h"
#include "mg.h"
#include "mg_slab.cuh"
#include "rmt3d_gpu.h"

namespace rmt3d {

template <typename T, int KIND, bool VD>
__global__ void __launch_bounds__(kSlabThreads, 1) k_mg_slab(const __grid_constant__ pmg_args A,
                                                           const __grid_constant__ slab_args S) {
    extern __shared__ __align__(16) unsigned char slab_smem[];
    slab_cycle<T, KIND, VD>(A, S, slab_smem);
}

// the same for every running scene of a group: cluster b works on scene b
template <typename T, int KIND, bool VD>
__global__ void __launch_bounds__(kSlabThreads, 1) k_mg_slab_b(const pmg_args *A, const int *run,
                                                             const __grid_constant__ slab_args S) {
    extern __shared__ __align__(16) unsigned char slab_smem[];
    const int b = blockIdx.x / S.csize;
    if (!run[b]) return;  // the whole cluster leaves together
    slab_cycle<T, KIND, VD>(A[b], S, slab_smem);
}

// ---- host side -------------------------------------------------------------
constexpr size_t kSlabSmemMax = 227 * 1024 - 1024;

namespace {
template <typename T>
const void *slab_fn(bool fem, bool vd, bool batched) {
    if (batched)
        return fem ? (vd ? (const void *)k_mg_slab_b<T, 1, true> : (const void *)k_mg_slab_b<T, 1, false>)
                   : (vd ? (const void *)k_mg_slab_b<T, 0, true> : (const void *)k_mg_slab_b<T, 0, false>);
    return fem ? (vd ? (const void *)k_mg_slab<T, 1, true> : (const void *)k_mg_slab<T, 1, false>)
               : (vd ? (const void *)k_mg_slab<T, 0, true> : (const void *)k_mg_slab<T, 0, false>);
}
const void *slab_fn(bool f32, bool fem, bool vd, bool batched) {
    return f32 ? slab_fn<float>(fem, vd, batched) : slab_fn<double>(fem, vd, batched);
}

cudaError_t slab_go(const void *fn, void **args, int clusters, int csize, size_t smem, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * csize);
    cfg.blockDim = dim3(kSlabThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = csize;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}
}  // namespace

// the kernels' attributes, the largest cluster whose CTAs fit this device with
// the largest shared memory (0: neither 16 nor 8), and how many such clusters
// run at once (once per device)
namespace {
struct slab_device {
    int size = 0, at_once = 0;
};
slab_device query_device() {
    slab_device q;
    for (int m = 0; m < 16; m++) {
        const void *fn = slab_fn(m & 1, m & 2, m & 4, m & 8);
        if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
            cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSlabSmemMax) != cudaSuccess) {
            cudaGetLastError();
            return q;
        }
    }
    for (int c : {16, 8}) {
        int least = 1 << 30;
        for (int m = 0; m < 16; m++) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(kSlabThreads);
            cfg.dynamicSmemBytes = kSlabSmemMax;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = c;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int n = 0;
            if (cudaOccupancyMaxActiveClusters(&n, slab_fn(m & 1, m & 2, m & 4, m & 8), &cfg) != cudaSuccess) {
                cudaGetLastError();
                n = 0;
            }
            least = std::min(least, n);
        }
        if (least >= 1) {
            q.size = c;
            q.at_once = least;
            break;
        }
    }
    return q;
}
slab_device this_device() {
    static std::mutex mu;
    static slab_device known[64];
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return slab_device();
    std::lock_guard<std::mutex> lk(mu);
    if (!done[dev]) known[dev] = query_device();
    done[dev] = true;
    return known[dev];
}
}  // namespace

int slab_cluster_size() { return this_device().size; }

// A group's clusters, one a scene, run in waves of as many as fit the device (7
// of 16 CTAs on a B200), while its per-phase launches fill the device with all
// scenes' points.  Against those, step time of groups of 12^3 to 96^3 scenes,
// both densities, FP64 and mixed: one wave 1.03 to 1.5 times as fast, two
// waves (8 to 14 scenes) 0.84 to 1.11, three (15) 0.73 to 0.99, five (32) 0.61
// to 0.91.
bool slab_pays(int scenes) { return scenes <= 2 * this_device().at_once; }

bool slab_fits(const mg_solver &m, int l0) {
    const size_t b = slab_layout(m.lv, l0, m.slab_csize, !m.mixed, m.vd, false, nullptr);
    return b > 0 && b <= kSlabSmemMax;
}

cudaError_t slab_cycle_launch(const mg_solver &m, int l0, bool f32, cudaStream_t st) {
    slab_args S;
    const size_t smem = slab_layout(m.lv, l0, m.slab_csize, !f32, m.vd, l0 == 0 && !f32, &S);
    pmg_args A = level_args(m);
    void *args[2] = {&A, &S};
    return slab_go(slab_fn(f32, m.kind == MG_FEM, m.vd, false), args, 1, S.csize, smem, st);
}

cudaError_t slab_cycle_launch_b(const mg_group &g, int l0, bool f32, cudaStream_t st) {
    slab_args S;
    const size_t smem = slab_layout(g.lv, l0, g.csize, !f32, g.vd, l0 == 0 && !f32, &S);
    const pmg_args *A = g.dargs;
    const int *run = g.run;
    void *args[3] = {(void *)&A, (void *)&run, &S};
    return slab_go(slab_fn(f32, g.kind == MG_FEM, g.vd, true), args, g.B, S.csize, smem, st);
}

}  // namespace rmt3d
