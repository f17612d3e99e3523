// cluster.cuh -- thread-block clusters: barriers and stores into the other blocks' shared memory.
#pragma once

#include <map>
#include <mutex>
#include <tuple>

#include "porsol_internal.h"

namespace porsol {

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// hardware barrier over all threads of the cluster: remote stores before it are visible after it
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync()
{
    cluster_arrive();
    cluster_wait();
}
// address of this block's shared location `a` in the block of rank r
__device__ __forceinline__ unsigned map_rank(unsigned a, unsigned r)
{
    unsigned d;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(r));
    return d;
}
__device__ __forceinline__ void put(unsigned a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void put(unsigned a, double v)
{
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

__device__ __forceinline__ void put(unsigned a, int v)
{
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Whether the current device can hold a cluster of `ctas` blocks of the kernel (more than 8 is opt-in, and a
// partition or a part with fewer SMs in each of its groups may hold fewer): asked once per device and shape.
// Leaves the kernel ready for a launch of that shape; callers have another way where the answer is no.
template <class... KA>
inline bool cluster_fits(void (*kernel)(KA...), int ctas, int threads, size_t shm)
{
    static std::mutex m;
    static std::map<std::tuple<int, const void*, int, int, size_t>, bool> known;
    int dev = 0;
    PORSOL_CUDA(cudaGetDevice(&dev));
    const auto key = std::make_tuple(dev, (const void*)kernel, ctas, threads, shm);
    std::lock_guard<std::mutex> lk(m);
    const auto it = known.find(key);
    if (it != known.end()) return it->second;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = ctas;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = shm;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    const bool fits =
        (shm <= 40 * 1024 ||   // static shared memory comes on top of it within the default 48 KB
         cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(shm)) == cudaSuccess) &&
        (ctas <= 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
    cudaGetLastError();
    return known[key] = fits;
}

// Launch of one cluster of `ctas` blocks, chained (chain()) when pdl.
template <class... KA, class... A>
inline void launch_cluster(void (*kernel)(KA...), int ctas, int threads, size_t shm, cudaStream_t s, bool pdl, A&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = ctas;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = shm;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 2 : 1;
    PORSOL_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...));
    PORSOL_COUNT_LAUNCH();
}

}  // namespace porsol
