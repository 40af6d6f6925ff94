// Prefill kernel instantiations for head sizes 192, 256.
#include "prefill_inst.cuh"

namespace b200pa {
PrefillKernelInfo find_prefill_large(int d, int q_dtype, int kv_dtype) {
  switch (d) {
    case 192: return find_prefill_for<192>(q_dtype, kv_dtype);
    case 256: return find_prefill_for<256>(q_dtype, kv_dtype);
  }
  return {nullptr, 0};
}
}  // namespace b200pa
