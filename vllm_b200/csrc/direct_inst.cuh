// Explicit-instantiation helper of the direct decode kernel (direct_*.cu).
#pragma once

#include "cluster_fit.h"
#include "decode_direct.cuh"

namespace b200pa {

using DirectLaunchFn = cudaError_t (*)(const DecodeParams&, int items, int cluster, cudaStream_t stream);

struct DirectKernelInfo {
  DirectLaunchFn fn;
  int ctas_per_sm;  // that the register budget is set for
  int resident;     // that fit in fact
};

template <typename QT, int KV, int D, int GP>
cudaError_t direct_launch(const DecodeParams& p, int items, int cluster, cudaStream_t stream) {
  auto kern = pa_decode_direct_kernel<QT, KV, D, GP>;
  constexpr int smem = DirectShape<KV, D, GP>::kSmem;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kDirectWarps * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  auto set_clusters = [&](int n, int size) {
    attr[1].val.clusterDim.x = size;
    cfg.gridDim = dim3(unsigned(n) * unsigned(size));
    cfg.numAttrs = size > 1 ? 2 : 1;
  };
  // once per device: opt in to clusters of 16 and (for wide heads) more than 48 KiB of shared memory, and
  // see what the device has room for
  static int largest[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int limit = dev >= 0 && dev < 64 ? largest[dev] : 0;
  if (limit == 0) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();
      return e;
    }
    (void)cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    limit = largest_cluster([&](int size) {
      set_clusters(1, size);
      int places = 0;
      return cudaOccupancyMaxActiveClusters(&places, kern, &cfg) == cudaSuccess ? places : 0;
    });
    (void)cudaGetLastError();  // (of sizes that the device refused)
    if (dev >= 0 && dev < 64) largest[dev] = limit;
  }
  if (cluster > limit) cluster = limit;
  set_clusters(items, cluster);
  return cudaLaunchKernelEx(&cfg, kern, p, cluster);
}

template <typename QT, int KV, int D>
DirectKernelInfo direct_gp(int gp) {
  using S1 = DirectShape<KV, D, 1>;
  if (gp == 1) return {direct_launch<QT, KV, D, 1>, S1::kMinCtas, S1::kResident};
  if constexpr (D <= 128) {
    using S2 = DirectShape<KV, D, 2>;
    return {direct_launch<QT, KV, D, 2>, S2::kMinCtas, S2::kResident};
  }
  return {nullptr, 0, 0};  // (two head tiles of a wide head do not fit the registers)
}

template <typename QT, int D>
DirectKernelInfo direct_kv(int kv_dtype, int gp) {
  if (kv_dtype == B200PA_KV_AUTO) return direct_gp<QT, kCache16, D>(gp);
  if constexpr (D % 16 == 0) {
    if (kv_dtype == B200PA_KV_FP8_E4M3) return direct_gp<QT, kCacheE4M3, D>(gp);
    if (kv_dtype == B200PA_KV_FP8_E5M2) return direct_gp<QT, kCacheE5M2, D>(gp);
  }
  return {nullptr, 0, 0};
}

// gp: 8-head tiles per work item (1 or 2)
template <int D>
DirectKernelInfo find_direct_for(int q_dtype, int kv_dtype, int gp) {
  if (q_dtype == B200PA_BF16) return direct_kv<__nv_bfloat16, D>(kv_dtype, gp);
  if (q_dtype == B200PA_F16) return direct_kv<__half, D>(kv_dtype, gp);
  return {nullptr, 0, 0};
}

// Defined in direct_small.cu (32 .. 96), direct_mid.cu (112 .. 128), direct_large.cu (192, 256).
DirectKernelInfo find_direct_small(int d, int q_dtype, int kv_dtype, int gp);
DirectKernelInfo find_direct_mid(int d, int q_dtype, int kv_dtype, int gp);
DirectKernelInfo find_direct_large(int d, int q_dtype, int kv_dtype, int gp);

}  // namespace b200pa
