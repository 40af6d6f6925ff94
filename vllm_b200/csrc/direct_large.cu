// Direct decode kernel instantiations for head sizes 192, 256.
#include "direct_inst.cuh"

namespace b200pa {
DirectKernelInfo find_direct_large(int d, int q_dtype, int kv_dtype, int gp) {
  switch (d) {
    case 192: return find_direct_for<192>(q_dtype, kv_dtype, gp);
    case 256: return find_direct_for<256>(q_dtype, kv_dtype, gp);
  }
  return {nullptr, 0};
}
}  // namespace b200pa
