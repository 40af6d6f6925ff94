// Prefill kernel instantiations for head sizes 32, 64, 80, 96.
#include "prefill_inst.cuh"

namespace b200pa {
PrefillKernelInfo find_prefill_small(int d, int q_dtype, int kv_dtype) {
  switch (d) {
    case 32: return find_prefill_for<32>(q_dtype, kv_dtype);
    case 64: return find_prefill_for<64>(q_dtype, kv_dtype);
    case 80: return find_prefill_for<80>(q_dtype, kv_dtype);
    case 96: return find_prefill_for<96>(q_dtype, kv_dtype);
  }
  return {nullptr, 0};
}
}  // namespace b200pa
