#include "launchers.h"
#include "step_reg.cuh"
namespace sqb {
template <int KIND, int BITS>
static int launch_reg_wide(const StepArgs& a, cudaStream_t stream) {
  return a.DV == 64 ? launch_reg_one<KIND, BITS, 128, 64, 2>(a, stream) : launch_reg_one<KIND, BITS, 128, 128, 1>(a, stream);
}
template <int BITS>
static int launch_reg_96(const StepArgs& a, cudaStream_t stream) {
  if (a.DV == 64) return launch_reg_one<K_GDN, BITS, 96, 64, 2>(a, stream);
  return a.DV == 128 ? launch_reg_one<K_GDN, BITS, 96, 128, 1>(a, stream) : launch_reg_one<K_GDN, BITS, 96, 192, 1>(a, stream);
}
int launch_reg(int kind, const StepArgs& a, int bits, cudaStream_t stream) {
  if (a.DK == 96) return bits == 8 ? launch_reg_96<8>(a, stream) : launch_reg_96<4>(a, stream);
  if (kind == K_GDN)
    return bits == 16 ? launch_reg_wide<K_GDN, 16>(a, stream) : bits == 8 ? launch_reg_wide<K_GDN, 8>(a, stream) : launch_reg_wide<K_GDN, 4>(a, stream);
  return bits == 16 ? launch_reg_wide<K_M2, 16>(a, stream) : bits == 8 ? launch_reg_wide<K_M2, 8>(a, stream) : launch_reg_wide<K_M2, 4>(a, stream);
}
}  // namespace sqb
