// Thread-block clusters: ranks, remote shared-memory stores, remote mbarrier arrivals.  Every spin is bounded.
#pragma once

#include <mutex>

#include "cq_ptx.cuh"

namespace cq {
namespace cluster {

using ptx::smem_u32;

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t cluster_size() { uint32_t r; asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t map_peer(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_peer(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void st_peer2(uint32_t addr, float a, float b) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(a), "f"(b) : "memory");
}
__device__ __forceinline__ void arrive_peer(uint32_t bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool wait_peers(uint64_t* bar, uint32_t max_tries) {      // phase 0, writes of the peers visible
#pragma unroll 1
  for (uint32_t i = 0; i < max_tries; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)) : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// ---- host: how many clusters of S CTAs (256 threads, two CTAs per SM) are resident at once.  Clusters do not straddle
// GPCs, whose SM counts differ from GPU to GPU: of 296 slots a B200 fills 296 / 148 / 71 / 33 clusters of 1 / 2 / 4 / 8.
// Asked of the runtime once per device and size.
static __global__ void __launch_bounds__(256, 2) residency_probe() {}
inline int max_clusters(int S) {
  static int known[64][9] = {};
  static std::mutex mu;
  const int fallback = S >= 8 ? 33 : S >= 4 ? 71 : S >= 2 ? 148 : 296;
  int dev = 0;
  if (S > 8 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { (void)cudaGetLastError(); return fallback; }
  std::lock_guard<std::mutex> lock(mu);
  int& n = known[dev][S];
  if (n == 0) {
    constexpr int SMEM = 104 * 1024;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(64 * S);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = SMEM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(residency_probe, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, residency_probe, &cfg) != cudaSuccess || n <= 0) {
      (void)cudaGetLastError();
      n = fallback;
    }
  }
  return n;
}

}  // namespace cluster
}  // namespace cq
