// sw_step.h -- host side of the whole-step kernel (sw_step.cuh): which tile
// shape a grid takes, and the launch.
#pragma once
#include "sw_step.cuh"

namespace swb {

// Tile shape (index into the shapes of sw_step.cu) and the tiles in x and y;
// shape < 0: the grid has no such plan.
struct StepPlan {
    int shape = -1, ntx = 0, nty = 0;
};

// hvar: the depth varies along x
template <class T>
StepPlan step_plan(const Geom& g, int nsm, bool hvar);
template <class T>
cudaError_t step_launch(const StepPlan& plan, StepArgs<T> a, bool hvar, cudaStream_t stream);

}  // namespace swb
