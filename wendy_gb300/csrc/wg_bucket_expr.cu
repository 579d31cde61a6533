// wg_bucket_expr.cu -- the fused sub-step for launches with expression forces
// (its instantiations carry the expression interpreter).
#include "wg_bucket_step.cuh"

namespace wg {

StepKernel step_kernel_expr(bool last, int mass) {
  if (mass == kMassAny)
    return last ? k_bucket_step<true, kForceExpr, kMassAny>
                : k_bucket_step<false, kForceExpr, kMassAny>;
  // equal masses are decided per task here
  return last ? k_bucket_step<true, kForceExpr, kMassMixed>
              : k_bucket_step<false, kForceExpr, kMassMixed>;
}

}  // namespace wg
