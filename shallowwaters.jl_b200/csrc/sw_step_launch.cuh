// sw_step_launch.cuh -- tile shapes of the whole-step kernel, their choice and
// the launch; instantiated for the RK schemes in sw_step.cu and for the SSP
// schemes in sw_step_ssp.cu.
#pragma once
#include <algorithm>
#include <array>
#include <cstdlib>

#include "sw_step.h"

namespace swb {
namespace {

// Tile shapes (StepShape: warps side by side, warps, rows per thread).  Low
// tiles for grids that leave SMs idle: a pass is then one row's latency, and
// more rows per block cost more clocks than their halos (Float32, us a step,
// 64x32: 20 rows 9.5, 24 10.0, 32 11.0; 256x128 needs 24 rows to run in one
// wave, 10.8 against 18.7).  32 rows fill the gap up to 512x256 (400x200: 13.5,
// else 15.7), 2 warps side by side the ones above (512x256: 20.0 against 22.5).
// The last shape fills the shared memory of an SM, for several waves
// (2048x1024: 137 against 170); with a depth that varies along x the eighth
// array costs it rows.
// 24 warps leave 80 registers a thread, which spills 16 to 84 bytes (164 in a
// batch); where that shape is picked the next one, which spills nothing, is
// slower all the same (256x128: 11.8 against 10.8, SSPRK3 128x64 15.5 against
// 13.8).
template <class T, bool HVAR>
struct Shapes;
template <bool HVAR>
struct Shapes<float, HVAR> {
    using S0 = StepShape<float, 1, 20, 1>;
    using S1 = StepShape<float, 1, 24, 1>;
    using S2 = StepShape<float, 1, 16, 2>;
    using S3 = StepShape<float, 2, 16, 4>;
    using S4 = StepShape<float, 2, 16, HVAR ? 7 : 8>;
};
template <bool HVAR>
struct Shapes<double, HVAR> {
    using S0 = StepShape<double, 1, 20, 1>;
    using S1 = StepShape<double, 1, 24, 1>;
    using S2 = StepShape<double, 1, 16, 2>;
    using S3 = StepShape<double, 1, 16, 4>;
    using S4 = StepShape<double, 2, 16, 7>;
};
constexpr int NSHAPES = 5;

// Tiles in x of shapes with cols columns; 0 if the grid has no split.
inline int split_cols(int N, int ep, int cols, int lo, int hi) {
    if (N + 4 <= cols) return 1;
    const int cap = cols - lo - hi, L = ep ? N + 8 : N;
    const int n = (L + cap - 1) / cap;
    // the second tile's halo must not reach across x = 0, nor the last but one's across x = N
    return L / n >= (lo > hi ? lo : hi) + 4 ? n : 0;
}

struct ShapeInfo { int cols, EWW, EH; };
template <class T, bool HVAR>
std::array<ShapeInfo, NSHAPES> shape_infos() {
    using SS = Shapes<T, HVAR>;
    auto of = [](auto s) {
        using S = decltype(s);
        return ShapeInfo{S::COLS, S::EWW, S::EH};
    };
    return {of(typename SS::S0{}), of(typename SS::S1{}), of(typename SS::S2{}), of(typename SS::S3{}), of(typename SS::S4{})};
}
// a tile's clocks: its passes' latencies and barriers, and its rows, measured.
// One line serves all forms, as only the order of the shapes matters: of the
// five forced in turn it picks the fastest (within 1 %) for Float32, Float64,
// SSPRK3, SSPRK2 with Sadourny in Float64 and bf16 storage at each of seven
// sizes from 64x32 to 2999x1499.
inline double tile_clocks(const ShapeInfo& f, int rows) { return 7000.0 + 540.0 * f.EWW * rows; }

template <class T, bool HVAR>
StepPlan plan_of(const Geom& g, int nsm, int lo, int hi) {
    const auto info = shape_infos<T, HVAR>();
    // forces a shape (and the rows per tile), or the launches per stage (-1)
    const char* env = getenv("SWB200_STEP");
    const char* envr = getenv("SWB200_STEP_ROWS");
    const int only = env ? atoi(env) : NSHAPES, rows = envr ? atoi(envr) : 0;
    StepPlan best;
    if (only < 0) return best;
    double cost = 1e30;
    for (int s = 0; s < NSHAPES; s++) {
        if (only < NSHAPES && s != only) continue;
        const ShapeInfo& f = info[s];
        const int ntx = split_cols(g.N, g.ep, f.cols, lo, hi);
        if (!ntx) continue;
        const int hmax = std::min(g.M + 4 <= f.EH ? g.M : f.EH - lo - hi, g.M);
        for (int h = hmax; h >= 2; h--) {
            const int nty = (g.M + h - 1) / h, hh = (g.M + nty - 1) / nty;
            if (g.M / nty < 2) continue;   // the wall tiles hold the sources of both ghost rows
            if (rows > 0 && nty != (g.M + std::min(rows, hmax) - 1) / std::min(rows, hmax)) continue;
            const int EHv = std::min(hh + lo + hi, g.M + 4);
            const int waves = (ntx * nty + nsm - 1) / nsm;
            const double c = waves * tile_clocks(f, EHv);
            if (c < cost) { cost = c; best = StepPlan{s, ntx, nty}; }
        }
    }
    return best;
}

// a launch that is prepared while the kernel before it runs; the kernel waits for that one's end
template <class S, class Kernel, class... Args>
cudaError_t go_prepared(Kernel kern, int smem, int nblocks, cudaStream_t stream, const Args&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = nblocks;
    cfg.blockDim = S::NW * 32;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// without arguments: allows the kernel its shared memory in the current CUDA context
template <class T, class S, bool HVAR, bool SSP, bool SAD>
cudaError_t go(const StepArgs<T>* a, cudaStream_t stream) {
    auto kern = rk_step_kernel<T, S, HVAR, SSP, SAD>;
    constexpr int smem = S::smem(HVAR);
    static_assert(smem <= 227 * 1024, "tile beyond the shared memory of an SM");
    if (!a) return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return go_prepared<S>(kern, smem, a->ntx * a->nty, stream, *a);
}

template <class T, bool HVAR, bool SSP, bool SAD>
cudaError_t go_shape(int shape, const StepArgs<T>* a, cudaStream_t stream) {
    using SS = Shapes<T, HVAR>;
    if (shape == 0) return go<T, typename SS::S0, HVAR, SSP, SAD>(a, stream);
    if (shape == 1) return go<T, typename SS::S1, HVAR, SSP, SAD>(a, stream);
    if (shape == 2) return go<T, typename SS::S2, HVAR, SSP, SAD>(a, stream);
    if (shape == 3) return go<T, typename SS::S3, HVAR, SSP, SAD>(a, stream);
    return go<T, typename SS::S4, HVAR, SSP, SAD>(a, stream);
}

}  // namespace

template <class T>
StepPlan step_plan(const Geom& g, int nsm, bool hvar, bool ssp) {
    const int lo = ssp ? STEP_LO_SSP : STEP_LO, hi = ssp ? STEP_HI_SSP : STEP_HI;
    return hvar ? plan_of<T, true>(g, nsm, lo, hi) : plan_of<T, false>(g, nsm, lo, hi);
}

template <class T, bool SSP>
void set_constants(StepArgs<T>& a) {
    using K = Pack<T>;
    a.lo = SSP ? STEP_LO_SSP : STEP_LO;
    a.hi = SSP ? STEP_HI_SSP : STEP_HI;
    a.half = K::host(T(0.5));
    a.q4 = K::host(T(0.25));
    a.o12 = K::host(T(1.0 / 12.0));
    a.nz = K::host(T(-0.0));
}

template <class T, bool SSP>
cudaError_t go_variant(int shape, const StepArgs<T>* a, bool hvar, bool sad, cudaStream_t stream) {
    if (hvar) return sad ? go_shape<T, true, SSP, true>(shape, a, stream) : go_shape<T, true, SSP, false>(shape, a, stream);
    return sad ? go_shape<T, false, SSP, true>(shape, a, stream) : go_shape<T, false, SSP, false>(shape, a, stream);
}

template <class T, bool SSP>
cudaError_t step_prepare(const StepPlan& p, bool hvar, bool sad) {
    return go_variant<T, SSP>(p.shape, nullptr, hvar, sad, nullptr);
}

template <class T, bool SSP>
cudaError_t step_launch(const StepPlan& p, StepArgs<T> a, bool hvar, bool sad, cudaStream_t stream) {
    a.ntx = p.ntx;
    a.nty = p.nty;
    set_constants<T, SSP>(a);
    return go_variant<T, SSP>(p.shape, &a, hvar, sad, stream);
}

}  // namespace swb
