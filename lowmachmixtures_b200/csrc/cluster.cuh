// cluster.cuh - thread-block clusters: barriers, stores into another block's
// shared memory, and the launch (with the programmatic dependence of pdl.cuh).
#pragma once
#include <cuda_runtime.h>

#include "stencil.cuh"

namespace lmm {

// every thread of every block arrives; the two halves of cluster_sync.  A block
// waits once for the others before its first store into their shared memory
// (they must have started) and leaves only after a barrier that follows the
// last store into its own.
__device__ __forceinline__ void cluster_arrive() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_sync() {
    cluster_arrive();
    cluster_wait();
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the address of shared-memory byte `a` of the block with rank r
__device__ __forceinline__ unsigned dsmem_at(unsigned a, unsigned r) {
    unsigned o;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(r));
    return o;
}
__device__ __forceinline__ void dsmem_store(unsigned a, float v) {
#ifdef LMM_BOUNDS_CHECK
    if (!bc_cluster_ok(a, sizeof(v))) return;
#endif
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void dsmem_store(unsigned a, double v) {
#ifdef LMM_BOUNDS_CHECK
    if (!bc_cluster_ok(a, sizeof(v))) return;
#endif
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// clusters of nc.x x nc.y x nc.z blocks, ranked x fastest (each extent of the grid a multiple of its)
template <class... KArgs, class... Args>
static inline cudaError_t launch_cluster(void (*k)(KArgs...), dim3 grid, dim3 block, dim3 nc, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = nc.x;
    at[1].val.clusterDim.y = nc.y;
    at[1].val.clusterDim.z = nc.z;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace lmm
