// Team kernel for k in (32, 64].
#include "team_kernel.cuh"

namespace lpgpu {

const void* team_kernel_w2(bool unit, int unroll, int minb) {
  return unit ? team_kernel_wu<2, true>(unroll, minb) : team_kernel_wu<2, false>(unroll, minb);
}

}  // namespace lpgpu
