// Thread-block-cluster primitives.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rmt3d {

// every thread of the cluster; orders shared and global memory
__device__ __forceinline__ void cl_barrier() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
}
__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// generic address, in CTA `rank` of the cluster, of what p is here
template <typename T>
__device__ __forceinline__ T *cl_map(T *p, unsigned rank) {
    T *q;
    asm("mapa.u64 %0, %1, %2;" : "=l"(q) : "l"(p), "r"(rank));
    return q;
}

// ---- values sent to a neighbour CTA ----------------------------------------
// A send stores a value into another CTA's shared memory and counts its bytes
// on an mbarrier there (st.async): value and signal travel together, with no
// fence.  The receiver arms a phase with the bytes it will get, and waits.
typedef unsigned cl_addr;  // shared::cluster address
template <typename T>
__device__ __forceinline__ cl_addr cl_remote(T *p, unsigned rank) {
    cl_addr a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cl_send(cl_addr a, float v, cl_addr bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];\n" ::"r"(a),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cl_send(cl_addr a, double v, cl_addr bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];\n" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void halo_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void halo_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void halo_arm(uint64_t *bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(bar)),
                 "r"(bytes)
                 : "memory");
}
// false if the phase did not complete within the limit (every send belongs to
// a pass the sender has begun, so this does not happen; the bound keeps a
// fault from turning into a hang; a wait takes 4 us, so about 4 s)
__device__ __forceinline__ bool halo_wait(uint64_t *bar, unsigned parity) {
    const unsigned b = (unsigned)__cvta_generic_to_shared(bar);
    for (int it = 0; it < (1 << 20); it++) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(b), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// about a millisecond, a thousand times what a send takes
__device__ __forceinline__ void cl_linger() {
    for (int it = 0; it < 16; it++) __nanosleep(64000);
}

}  // namespace rmt3d
