// sw_step.cu -- the whole-step kernel for the RK schemes.
#include "sw_step_launch.cuh"

namespace swb {
template StepPlan step_plan<float>(const Geom&, int, bool, bool);
template StepPlan step_plan<double>(const Geom&, int, bool, bool);
template cudaError_t step_prepare<float, false>(const StepPlan&, bool, bool);
template cudaError_t step_prepare<double, false>(const StepPlan&, bool, bool);
template cudaError_t step_launch<float, false>(const StepPlan&, StepArgs<float>, bool, bool, cudaStream_t);
template cudaError_t step_launch<double, false>(const StepPlan&, StepArgs<double>, bool, bool, cudaStream_t);
}  // namespace swb
