// sw_step_ssp.cu -- the whole-step kernel for the SSP schemes.
#include "sw_step_launch.cuh"

namespace swb {
template cudaError_t step_prepare<float, true>(const StepPlan&, bool, bool);
template cudaError_t step_prepare<double, true>(const StepPlan&, bool, bool);
template cudaError_t step_launch<float, true>(const StepPlan&, StepArgs<float>, bool, bool, cudaStream_t);
template cudaError_t step_launch<double, true>(const StepPlan&, StepArgs<double>, bool, bool, cudaStream_t);
}  // namespace swb
