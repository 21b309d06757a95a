// Instantiations of the fused step kernel: double, spin1 model.
#include "fused_impl.cuh"

namespace clv {
void *fused_kernel_f64_spin1(int ln, bool fast, bool two) { return fused_fn<double, CLV_MODEL_SPIN1, true>(ln, fast, two); }
}  // namespace clv
