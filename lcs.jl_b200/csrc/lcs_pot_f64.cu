// Kernels of the couple in potential form in F64.  Built with --fmad=false, as the FP64
// engine is: what is to be contracted says so.
#include "lcs_potential.cuh"

namespace lcs {
const PotKernels<double>& pot_kernels_f64() {
  static const PotKernels<double> k = make_pot_kernels<double>();
  return k;
}
}  // namespace lcs
