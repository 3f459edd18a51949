// sw_step_s16.cu -- the whole-step kernel for the 16-bit storage form: the
// tiles of sw_step.cuh with Float32 arithmetic, the state read and written as
// pairs (Step16).  The stage increments, which the launches per stage keep in
// memory as 16-bit arrays, are rounded to that form and stay in the tile.
// us per step with the tracer beside it (B200, bf16; the launches per stage,
// then this): 64x32 70 and 11.2, 512x256 76 and 23.3, 1024x512 95 and 50.9,
// 2048x1024 308 and 169.  Its tallest tiles spill (8 rows 120 bytes in bf16 and
// 84 in half, 7 rows 80) and are the faster ones all the same: 2048x1024 takes
// 198 us in the next shape, which spills nothing.
#include "sw_step_launch.cuh"

namespace swb {
namespace {

template <class SH, bool HVAR, class E>
__global__ void __launch_bounds__(SH::NW * 32, 1)
s16_step_kernel(const __grid_constant__ StepArgs<float> A, const __grid_constant__ Step16<E> io) {
    extern __shared__ __align__(16) unsigned char step_smem[];
    cudaTriggerProgrammaticLaunchCompletion();
    step_block<float, SH, HVAR, false, false>(A, (int)blockIdx.x, reinterpret_cast<typename SH::P*>(step_smem), io);
}

template <class SH, bool HVAR, class E>
cudaError_t go16(const StepArgs<float>* a, const Step16<E>& io, cudaStream_t stream) {
    auto kern = s16_step_kernel<SH, HVAR, E>;
    constexpr int smem = SH::smem(HVAR);
    if (!a) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return go_prepared<SH>(kern, smem, a->ntx * a->nty, stream, *a, io);
}

template <bool HVAR, class E>
cudaError_t go16_shape(int shape, const StepArgs<float>* a, const Step16<E>& io, cudaStream_t stream) {
    using SS = Shapes<float, HVAR>;
    if (shape == 0) return go16<typename SS::S0, HVAR>(a, io, stream);
    if (shape == 1) return go16<typename SS::S1, HVAR>(a, io, stream);
    if (shape == 2) return go16<typename SS::S2, HVAR>(a, io, stream);
    if (shape == 3) return go16<typename SS::S3, HVAR>(a, io, stream);
    return go16<typename SS::S4, HVAR>(a, io, stream);
}

}  // namespace

template <class E>
cudaError_t step16_launch(const StepPlan& p, StepArgs<float> a, const Step16<E>& io, bool hvar, cudaStream_t stream) {
    a.ntx = p.ntx;
    a.nty = p.nty;
    set_constants<float, false>(a);
    return hvar ? go16_shape<true>(p.shape, &a, io, stream) : go16_shape<false>(p.shape, &a, io, stream);
}

template <class E>
cudaError_t step16_prepare(const StepPlan& p, bool hvar) {
    const Step16<E> io{};
    return hvar ? go16_shape<true>(p.shape, nullptr, io, nullptr) : go16_shape<false>(p.shape, nullptr, io, nullptr);
}

template cudaError_t step16_prepare<__nv_bfloat16>(const StepPlan&, bool);
template cudaError_t step16_prepare<__half>(const StepPlan&, bool);

template cudaError_t step16_launch(const StepPlan&, StepArgs<float>, const Step16<__nv_bfloat16>&, bool, cudaStream_t);
template cudaError_t step16_launch(const StepPlan&, StepArgs<float>, const Step16<__half>&, bool, cudaStream_t);

}  // namespace swb
