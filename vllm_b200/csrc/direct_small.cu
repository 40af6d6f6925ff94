// Direct decode kernel instantiations for head sizes 32, 64, 80, 96.
#include "direct_inst.cuh"

namespace b200pa {
DirectKernelInfo find_direct_small(int d, int q_dtype, int kv_dtype, int gp) {
  switch (d) {
    case 32: return find_direct_for<32>(q_dtype, kv_dtype, gp);
    case 64: return find_direct_for<64>(q_dtype, kv_dtype, gp);
    case 80: return find_direct_for<80>(q_dtype, kv_dtype, gp);
    case 96: return find_direct_for<96>(q_dtype, kv_dtype, gp);
  }
  return {nullptr, 0};
}
}  // namespace b200pa
