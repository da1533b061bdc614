#include "launchers.h"
#include "step_reg.cuh"
namespace sqb {
int launch_reg(int kind, const StepArgs& a, int bits, cudaStream_t stream) {
  if (bits == 16) {
    if (kind == K_GDN) return a.DV == 64 ? launch_reg_one<K_GDN, 16, 128, 64, 2>(a, stream) : launch_reg_one<K_GDN, 16, 128, 128, 1>(a, stream);
    return a.DV == 64 ? launch_reg_one<K_M2, 16, 128, 64, 2>(a, stream) : launch_reg_one<K_M2, 16, 128, 128, 1>(a, stream);
  }
  if (bits == 8) {
    if (a.DV == 64) return launch_reg_one<K_GDN, 8, 96, 64, 2>(a, stream);
    return a.DV == 128 ? launch_reg_one<K_GDN, 8, 96, 128, 1>(a, stream) : launch_reg_one<K_GDN, 8, 96, 192, 1>(a, stream);
  }
  if (a.DV == 64) return launch_reg_one<K_GDN, 4, 96, 64, 2>(a, stream);
  return a.DV == 128 ? launch_reg_one<K_GDN, 4, 96, 128, 1>(a, stream) : launch_reg_one<K_GDN, 4, 96, 192, 1>(a, stream);
}
}  // namespace sqb
