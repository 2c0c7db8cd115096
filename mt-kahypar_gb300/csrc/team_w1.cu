// Team kernel for k <= 32.
#include "team_kernel.cuh"

namespace lpgpu {

const void* team_kernel_w1(bool unit, int unroll, int minb) {
  return unit ? team_kernel_wu<1, true>(unroll, minb) : team_kernel_wu<1, false>(unroll, minb);
}

}  // namespace lpgpu
