// Team kernel for k in (256, 512].
#include "team_kernel.cuh"

namespace lpgpu {

const void* team_kernel_w16(bool unit, int unroll, int minb) {
  return unit ? team_kernel_wu<16, true>(unroll, minb) : team_kernel_wu<16, false>(unroll, minb);
}

}  // namespace lpgpu
