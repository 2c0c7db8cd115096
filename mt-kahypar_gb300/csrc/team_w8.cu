// Team kernel for k in (128, 256].
#include "team_kernel.cuh"

namespace lpgpu {

const void* team_kernel_w8(bool unit, int unroll, int minb) {
  return unit ? team_kernel_wu<8, true>(unroll, minb) : team_kernel_wu<8, false>(unroll, minb);
}

}  // namespace lpgpu
