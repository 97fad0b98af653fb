// rc_cluster.cuh -- CTAs of one thread-block cluster: rank, barrier, and stores to each other's shared memory.
#pragma once
#include <cstdint>

namespace rcb {

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
template <bool CL>
__device__ __forceinline__ void cl_sync() {
    if constexpr (CL) {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        __syncthreads();
    }
}
// The shared::cluster address of `p` in CTA `rank`, and stores to such addresses.
__device__ __forceinline__ uint32_t cl_addr(const void* p, unsigned rank) {
    uint32_t o;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return o;
}
__device__ __forceinline__ void cl_store(uint32_t a, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void cl_store(uint32_t a, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}

}  // namespace rcb
