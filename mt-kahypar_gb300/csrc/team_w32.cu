// Team kernel for k in (512, 1024].
#include "team_kernel.cuh"

namespace lpgpu {

const void* team_kernel_w32(bool unit, int unroll, int minb) {
  return unit ? team_kernel_wu<32, true>(unroll, minb) : team_kernel_wu<32, false>(unroll, minb);
}

}  // namespace lpgpu
