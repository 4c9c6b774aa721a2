// What the CTA-pair kernels share: the cta_group::2 forms of the PTX wrappers, the tensor map over stored shared-memory images
// and the number of pairs that can be resident. A pair is a cluster of two CTAs on neighbouring SMs; no load here is a
// multicast load.
#pragma once
#include "tc_host.cuh"
#include "tc_ptx.cuh"

namespace b200moe {

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// the shared::cluster address of `addr` (a shared::cta address of this CTA) in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_cta(uint32_t addr, uint32_t rank) {
  uint32_t out;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(out) : "r"(addr), "r"(rank));
  return out;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  // (release at CTA scope: what the arrival orders is tensor-memory reads, which tcgen05.wait::ld has completed; the cluster-scope
  // form also waits for the thread's global stores, 1300 cycles measured)
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// 2-D tile load whose bytes are counted on a barrier that may sit in the partner CTA (`bar` is a shared::cluster address)
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
          "r"(dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(cluster_addr) : "memory");
}
// the same, arriving on the barrier at this offset in both CTAs of the pair: one instruction (60 cycles of the thread) less
__device__ __forceinline__ void tc_commit_both(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
               "h"(static_cast<uint16_t>(3))
               : "memory");
}
__device__ __forceinline__ void tc_cp_scales_pair(uint32_t taddr, uint32_t desc_lo) {
  asm volatile("{\n.reg .b64 d;\nmov.b64 d, {%1, %2};\ntcgen05.cp.cta_group::2.32x128b.warpx4 [%0], d;\n}\n" ::"r"(taddr),
               "r"(desc_lo), "n"(kScaleDescHi)
               : "memory");
}
__device__ __forceinline__ void drain_tcgen05_pair(uint32_t bar) {
  tc_commit_pair(bar);
  const uint64_t t0 = global_timer(), limit = wait_limit_ns();
  while (!mbar_try_wait(bar, 0) && global_timer() - t0 < limit) {}
}

// ------------------------------------------------------------------------------------------------ host side
// byte matrix [rows][128], boxes of 128 bytes x box_rows, no swizzle (the bytes are stored as shared memory wants them)
static inline int make_flat_map(CUtensorMap* map, const void* base, uint64_t rows, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return B200MOE_E_DRIVER;
  const cuuint64_t dims[2] = {128, rows};
  const cuuint64_t strides[1] = {128};
  const cuuint32_t box[2] = {128, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : B200MOE_E_DRIVER;
}

// Pairs of `kernel` that can be resident at once on the current device (0: cluster launch unavailable); asked once per device
// and kernel (`known` and `pairs` are the kernel's own arrays of kMaxDevices, `mu` their lock).
template <typename K>
static inline int resident_pairs_of(K kernel, int threads, int smem, std::mutex& mu, bool* known, int* pairs) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 0;
  std::lock_guard<std::mutex> lock(mu);
  if (!known[dev]) {
    int n = 0;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(2 * sm_count());
      cfg.blockDim = dim3(threads);
      cfg.dynamicSmemBytes = smem;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) n = 0;
    }
    (void)cudaGetLastError();
    pairs[dev] = n;
    known[dev] = true;
  }
  return pairs[dev];
}

// Launches `clusters` CTA pairs with programmatic stream serialisation.
template <typename... KArgs, typename... Args>
static inline int launch_pairs(void (*kernel)(KArgs...), int clusters, int threads, int smem, cudaStream_t stream,
                               Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
  return e == cudaSuccess ? 0 : static_cast<int>(e);
}

}  // namespace b200moe
