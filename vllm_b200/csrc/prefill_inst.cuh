// Explicit-instantiation helper of the prefill kernel: each prefill_*.cu file builds it for some
// head sizes so that the files compile in parallel.
#pragma once

#include "prefill_kernel.cuh"

namespace b200pa {

using PrefillLaunchFn = cudaError_t (*)(const PrefillParams&, int grid, cudaStream_t stream);

struct PrefillKernelInfo {
  PrefillLaunchFn fn;
  int piece_bytes;  // workspace of one piece of an item
};

// Tensor maps.  V of a 16-bit cache: [block][kv head][D][block_size], boxes of 16 keys x D.  The number
// of blocks is not known here: block ids are taken as they come, as everywhere.  Q: [token][head][D],
// boxes of `box` head dimensions x the heads of a group x the tokens of a row tile.  Defined in
// varlen_attention.cu.
cudaError_t prefill_v_map(const PrefillParams& p, int head_size, CUtensorMap* map);
cudaError_t prefill_q_map(const PrefillParams& p, int head_size, int box, CUtensorMap* map);

template <typename QT, int KV, int D>
cudaError_t prefill_launch(const PrefillParams& p, int grid, cudaStream_t stream) {
  auto kern = pa_prefill_kernel<QT, KV, D>;
  constexpr int smem = PrefillShape<D>::kSmem;
  // opt in to large dynamic shared memory once per device
  static bool done[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64 || !done[dev]) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();  // do not leave the error for the next caller
      return e;
    }
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  CUtensorMap qmap, vmap = {};
  e = prefill_q_map(p, D, PrefillShape<D>::kQBox, &qmap);
  if (KV == kCache16 && e == cudaSuccess) e = prefill_v_map(p, D, &vmap);
  if (e != cudaSuccess) return e;
  return launch_dependent(kern, dim3(grid), dim3(kPrefillThreads), smem, stream, p, qmap, vmap);
}

template <typename QT, int D>
PrefillKernelInfo find_prefill_kv(int kv_dtype) {
  constexpr int piece = PrefillShape<D>::NQ * 128 * (D * 2 + 8);
  if (kv_dtype == B200PA_KV_AUTO) return {prefill_launch<QT, kCache16, D>, piece};
  if constexpr (D % 16 == 0) {
    if (kv_dtype == B200PA_KV_FP8_E4M3) return {prefill_launch<QT, kCacheE4M3, D>, piece};
    if (kv_dtype == B200PA_KV_FP8_E5M2) return {prefill_launch<QT, kCacheE5M2, D>, piece};
  }
  return {nullptr, 0};
}

template <int D>
PrefillKernelInfo find_prefill_for(int q_dtype, int kv_dtype) {
  if (q_dtype == B200PA_BF16) return find_prefill_kv<__nv_bfloat16, D>(kv_dtype);
  if (q_dtype == B200PA_F16) return find_prefill_kv<__half, D>(kv_dtype);
  return {nullptr, 0};
}

// Defined in prefill_small.cu (32 .. 96), prefill_mid.cu (112 .. 128), prefill_large.cu (192, 256).
PrefillKernelInfo find_prefill_small(int d, int q_dtype, int kv_dtype);
PrefillKernelInfo find_prefill_mid(int d, int q_dtype, int kv_dtype);
PrefillKernelInfo find_prefill_large(int d, int q_dtype, int kv_dtype);

}  // namespace b200pa
