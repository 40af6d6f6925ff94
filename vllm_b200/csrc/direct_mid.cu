// Direct decode kernel instantiations for head sizes 112, 120, 128.
#include "direct_inst.cuh"

namespace b200pa {
DirectKernelInfo find_direct_mid(int d, int q_dtype, int kv_dtype, int gp) {
  switch (d) {
    case 112: return find_direct_for<112>(q_dtype, kv_dtype, gp);
    case 120: return find_direct_for<120>(q_dtype, kv_dtype, gp);
    case 128: return find_direct_for<128>(q_dtype, kv_dtype, gp);
  }
  return {nullptr, 0};
}
}  // namespace b200pa
