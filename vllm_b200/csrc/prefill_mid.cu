// Prefill kernel instantiations for head sizes 112, 120, 128.
#include "prefill_inst.cuh"

namespace b200pa {
PrefillKernelInfo find_prefill_mid(int d, int q_dtype, int kv_dtype) {
  switch (d) {
    case 112: return find_prefill_for<112>(q_dtype, kv_dtype);
    case 120: return find_prefill_for<120>(q_dtype, kv_dtype);
    case 128: return find_prefill_for<128>(q_dtype, kv_dtype);
  }
  return {nullptr, 0};
}
}  // namespace b200pa
