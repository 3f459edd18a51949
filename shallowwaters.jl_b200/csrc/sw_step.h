// sw_step.h -- host side of the whole-step kernel (sw_step.cuh): which tile
// shape a grid takes, and the launch.
#pragma once
#include "sw_step.cuh"

namespace swb {

// Tile shape (index into the shapes of sw_step_launch.cuh) and the tiles in x
// and y; shape < 0: the grid has no such plan.
struct StepPlan {
    int shape = -1, ntx = 0, nty = 0;
};

// hvar: the depth varies along x; ssp: sub-stages of an SSP scheme
template <class T>
StepPlan step_plan(const Geom& g, int nsm, bool hvar, bool ssp);
// Allows the plan's kernel its shared memory, a setting of the current device
// and CUDA context: once per context before its first launch (the same for
// step16_prepare and step_batch_prepare).
template <class T, bool SSP>
cudaError_t step_prepare(const StepPlan& plan, bool hvar, bool sad);
// One step (sad: PV_Sadourny!); the arguments' tiles, halo and fixed constants are set here.
template <class T, bool SSP>
cudaError_t step_launch(const StepPlan& plan, StepArgs<T> a, bool hvar, bool sad, cudaStream_t stream);

// One step of the 16-bit storage form (Float32 arithmetic, RK, Arakawa-Hsu).
template <class E>
cudaError_t step16_prepare(const StepPlan& plan, bool hvar);
template <class E>
cudaError_t step16_launch(const StepPlan& plan, StepArgs<float> a, const Step16<E>& io, bool hvar, cudaStream_t stream);

// A launch over the tiles of up to STEP_BATCH members of an ensemble (Float32,
// RK, Arakawa-Hsu): members' arguments with their tiles (ntx, nty), their
// numbers of steps and the global step to run.
constexpr int STEP_BATCH = 64;
struct StepBatch {
    int n;
    int block0[STEP_BATCH + 1];        // set at the launch
    long long nt[STEP_BATCH];
    const long long* istep;
    StepArgs<float> m[STEP_BATCH];
};
static_assert(sizeof(StepBatch) <= 32764, "kernel parameters");
// The tile shape for members of these sizes and each member's tiles; -1: none.
int step_batch_plan(const Geom* gs, int n, int nsm, StepPlan* plans);
cudaError_t step_batch_prepare(int shape);
cudaError_t step_batch_launch(int shape, StepBatch& b, cudaStream_t stream);

}  // namespace swb
