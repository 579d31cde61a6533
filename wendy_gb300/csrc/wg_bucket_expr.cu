// wg_bucket_expr.cu -- the fused sub-step for launches with expression forces
// (its instantiations carry the expression interpreter; compiled apart from
// the others, beside them in time).
#include "wg_bucket_step.cuh"

namespace wg {

StepKernel step_kernel_expr(bool last, int mass) {
  if (mass == kMassAny)
    return last ? k_bucket_step<true, true, kMassAny> : k_bucket_step<false, true, kMassAny>;
  // equal masses are decided per task here
  return last ? k_bucket_step<true, true, kMassMixed> : k_bucket_step<false, true, kMassMixed>;
}

}  // namespace wg
