// Thread-block clusters: stores into another CTA's shared memory that complete
// on its mbarrier, the cluster barrier, and launches of 512-thread clusters.
#pragma once
#include "common.cuh"

namespace casphy {
namespace clu {

constexpr int kThreads = 512;  // of every cluster kernel
constexpr u32 kMaxG = 16;      // CTAs of a cluster (above 8 needs the opt-in placeable() makes)

__device__ __forceinline__ u32 smem_u32(const void* p) { return static_cast<u32>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ u32 mapa(u32 a, u32 rank) {
    u32 r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// Stores to a CTA of the cluster that complete on an mbarrier of the same CTA.
__device__ __forceinline__ void st_async16(u32 addr, uint4 r, u32 bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "r"(r.x), "r"(r.y), "r"(r.z), "r"(r.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async8(u32 addr, u64 v, u32 bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(u32 bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(u32 bar, u32 bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(u32 bar, u32 parity) {
    u32 ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0u;
}
// Waits for the phase; gives up after limitNs (recording CASPHY_ETIMEOUT) or
// when *err is set, and returns false.
__device__ __forceinline__ bool mbar_wait(u32 bar, u32 parity, int* err, u64 limitNs) {
    if (mbar_try(bar, parity)) return true;
    const u64 t0 = globaltimer_ns();
    while (!mbar_try(bar, parity)) {
        if (*(volatile int*)err) return false;
        if (globaltimer_ns() - t0 > limitNs) {
            atomicCAS(err, 0, CASPHY_ETIMEOUT);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ u32 cluster_rank() {
    u32 r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// Host: how many clusters of G CTAs of kernel fn the device can hold at once.
inline int placeable(void* fn, u32 G, size_t smem) {
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, fn, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// Host: queues `clusters` clusters of G CTAs of kernel fn(args...).
template <class... K, class... A>
cudaError_t enqueue(void (*fn)(K...), u32 G, u32 clusters, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G * clusters);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = G;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

// Host: one cluster; *done is false when the device cannot place it (nothing
// is launched then).
template <class... K, class... A>
int launch(void (*fn)(K...), u32 G, size_t smem, cudaStream_t st, bool* done, const A&... args) {
    *done = false;
    if (!placeable((void*)fn, G, smem)) return CASPHY_OK;
    CASPHY_CUDA_TRY(enqueue(fn, G, 1, smem, st, args...));
    *done = true;
    return CASPHY_OK;
}

}  // namespace clu
}  // namespace casphy
