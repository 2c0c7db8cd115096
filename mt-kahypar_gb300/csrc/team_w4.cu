// Team kernel for k in (64, 128].
#include "team_kernel.cuh"

namespace lpgpu {

const void* team_kernel_w4(bool unit, int unroll, int minb) {
  return unit ? team_kernel_wu<4, true>(unroll, minb) : team_kernel_wu<4, false>(unroll, minb);
}

}  // namespace lpgpu
