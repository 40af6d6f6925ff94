// Host side of tensor maps (cp.async.bulk.tensor): encoding through the driver's entry point, so that
// nothing has to be linked.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace b200pa {

// A tensor map of 16-bit elements without interleaving; `strides` in elements.  (L2 fetches 256 bytes at a time:
// large KV writes 1 to 2 % less than with 128, attention the same.)
template <int N>
inline cudaError_t tensor_map(CUtensorMap* map, const void* base, const int64_t (&dims)[N], const int64_t (&strides)[N - 1],
                              const int (&box)[N], CUtensorMapSwizzle swizzle) {
  using Encode = decltype(&cuTensorMapEncodeTiled);
  static const Encode encode = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<Encode>(f);
  }();
  if (encode == nullptr) return cudaErrorNotSupported;
  cuuint64_t d[N], st[N - 1];
  cuuint32_t b[N], step[N];
  for (int i = 0; i < N; ++i) {
    d[i] = cuuint64_t(dims[i]);
    b[i] = cuuint32_t(box[i]);
    step[i] = 1;
  }
  for (int i = 0; i < N - 1; ++i) st[i] = cuuint64_t(strides[i]) * 2;
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, N, const_cast<void*>(base), d, st, b, step,
                            CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Strides of 2-byte elements that a map can hold: positive, below 2^40 bytes (and multiples of 16 bytes).
inline bool tensor_map_stride(int64_t v) { return v > 0 && v < (int64_t(1) << 39); }

}  // namespace b200pa
