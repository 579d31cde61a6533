// wg_bucket_closed.cu -- the fused sub-step for launches with closed-form
// external forces.
#include "wg_bucket_step.cuh"

namespace wg {

StepKernel step_kernel_closed(bool last, int mass) {
  if (mass == kMassAny)
    return last ? k_bucket_step<true, kForceClosed, kMassAny> : k_bucket_step<false, kForceClosed, kMassAny>;
  if (mass == kMassEqual)
    return last ? k_bucket_step<true, kForceClosed, kMassEqual> : k_bucket_step<false, kForceClosed, kMassEqual>;
  return last ? k_bucket_step<true, kForceClosed, kMassMixed> : k_bucket_step<false, kForceClosed, kMassMixed>;
}

}  // namespace wg
