// cluster.cuh -- thread-block cluster helpers (rank, barrier, shared memory of
// the other CTAs).  A launch without the cluster attribute is a cluster of one.
#pragma once
#include <stdint.h>

namespace gbgpu {

__device__ __forceinline__ int cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ int cluster_size() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return (int)r;
}
// all threads of all CTAs of the cluster; orders their shared and global accesses
__device__ __forceinline__ void cluster_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of this CTA's shared object `p` in CTA `rank`
__device__ __forceinline__ uint32_t remote_smem(const void* p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(a)
                 : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ uint32_t remote_ld(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void remote_st(uint32_t a, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void remote_st4(uint32_t a, uint4 v) {
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w)
                 : "memory");
}

}  // namespace gbgpu
