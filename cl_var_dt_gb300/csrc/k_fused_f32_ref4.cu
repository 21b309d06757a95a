// Instantiations of the fused step kernel: float, ref4 model.
#include "fused_impl.cuh"

namespace clv {
void *fused_kernel_f32_ref4(int ln, bool fast) { return fused_fn<float, CLV_MODEL_REF4>(ln, fast); }
}  // namespace clv
