// Kernels of the couple in potential form in F32.  FMA contraction is allowed, as in the
// FP32 engine.
#include "lcs_potential.cuh"

namespace lcs {
const PotKernels<float>& pot_kernels_f32() {
  static const PotKernels<float> k = make_pot_kernels<float>();
  return k;
}
}  // namespace lcs
