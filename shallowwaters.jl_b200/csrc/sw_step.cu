// sw_step.cu -- instantiations of the whole-step kernel and the choice of its
// tile shape.
#include <algorithm>
#include <cstdlib>

#include "sw_step.h"

namespace swb {
namespace {

// Tile shapes (StepShape: warps side by side, warps, rows per thread, rows).
// Shape 2 fills the shared memory of an SM; with a depth that varies along x
// the eighth array costs it rows.
template <class T, bool HVAR>
struct Shapes;
template <bool HVAR>
struct Shapes<float, HVAR> {
    using S0 = StepShape<float, 1, 32, 1>;
    using S1 = StepShape<float, 2, 16, 4>;
    using S2 = StepShape<float, 2, 16, HVAR ? 7 : 8>;
};
template <bool HVAR>
struct Shapes<double, HVAR> {
    using S0 = StepShape<double, 1, 16, 2>;
    using S1 = StepShape<double, 1, 16, 4>;
    using S2 = StepShape<double, 2, 16, 7>;
};
constexpr int NSHAPES = 3;

// Tiles in x of shapes with cols columns; 0 if the grid has no split.
int split_cols(int N, int ep, int cols) {
    if (N + 4 <= cols) return 1;
    const int cap = cols - STEP_LO - STEP_HI, L = ep ? N + 8 : N;
    const int n = (L + cap - 1) / cap;
    // the second tile's halo must not reach across x = 0, nor the last but one's across x = N
    return L / n >= STEP_LO + 4 ? n : 0;
}

template <class T, bool HVAR>
StepPlan plan_of(const Geom& g, int nsm) {
    using SS = Shapes<T, HVAR>;
    struct Info { int cols, EWW, EH; };
    auto of = [](auto s) {
        using S = decltype(s);
        return Info{S::COLS, S::EWW, S::EH};
    };
    const Info info[NSHAPES] = {of(typename SS::S0{}), of(typename SS::S1{}), of(typename SS::S2{})};
    // forces a shape (and the rows per tile), or the launches per stage (-1)
    const char* env = getenv("SWB200_STEP");
    const char* envr = getenv("SWB200_STEP_ROWS");
    const int only = env ? atoi(env) : NSHAPES, rows = envr ? atoi(envr) : 0;
    StepPlan best;
    if (only < 0) return best;
    double cost = 1e30;
    for (int s = 0; s < NSHAPES; s++) {
        if (only < NSHAPES && s != only) continue;
        const Info& f = info[s];
        const int ntx = split_cols(g.N, g.ep, f.cols);
        if (!ntx) continue;
        const int hmax = std::min(g.M + 4 <= f.EH ? g.M : f.EH - STEP_LO - STEP_HI, g.M);
        for (int h = hmax; h >= 2; h--) {
            const int nty = (g.M + h - 1) / h, hh = (g.M + nty - 1) / nty;
            if (g.M / nty < 2) continue;   // the wall tiles hold the sources of both ghost rows
            if (rows > 0 && nty != (g.M + std::min(rows, hmax) - 1) / std::min(rows, hmax)) continue;
            const int EHv = std::min(hh + STEP_LO + STEP_HI, g.M + 4);
            const int waves = (ntx * nty + nsm - 1) / nsm;
            // a tile's clocks: its passes' latencies and barriers, and its rows, measured
            const double c = (double)waves * (7000.0 + 540.0 * f.EWW * EHv);
            if (c < cost) { cost = c; best = StepPlan{s, ntx, nty}; }
        }
    }
    return best;
}

template <class T, class S, bool HVAR>
cudaError_t go(const StepArgs<T>& a, cudaStream_t stream) {
    auto kern = rk_step_kernel<T, S, HVAR>;
    constexpr int smem = S::smem(HVAR);
    static_assert(smem <= 227 * 1024, "tile beyond the shared memory of an SM");
    static const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    kern<<<a.ntx * a.nty, S::NW * 32, smem, stream>>>(a);
    return cudaGetLastError();
}

template <class T, bool HVAR>
cudaError_t go_shape(int shape, const StepArgs<T>& a, cudaStream_t stream) {
    using SS = Shapes<T, HVAR>;
    if (shape == 0) return go<T, typename SS::S0, HVAR>(a, stream);
    if (shape == 1) return go<T, typename SS::S1, HVAR>(a, stream);
    return go<T, typename SS::S2, HVAR>(a, stream);
}

}  // namespace

template <class T>
StepPlan step_plan(const Geom& g, int nsm, bool hvar) {
    return hvar ? plan_of<T, true>(g, nsm) : plan_of<T, false>(g, nsm);
}

template <class T>
cudaError_t step_launch(const StepPlan& p, StepArgs<T> a, bool hvar, cudaStream_t stream) {
    a.ntx = p.ntx;
    a.nty = p.nty;
    a.half = Pack<T>::host(T(0.5));
    a.q4 = Pack<T>::host(T(0.25));
    a.o12 = Pack<T>::host(T(1.0 / 12.0));
    a.nz = Pack<T>::host(T(-0.0));
    return hvar ? go_shape<T, true>(p.shape, a, stream) : go_shape<T, false>(p.shape, a, stream);
}

template StepPlan step_plan<float>(const Geom&, int, bool);
template StepPlan step_plan<double>(const Geom&, int, bool);
template cudaError_t step_launch<float>(const StepPlan&, StepArgs<float>, bool, cudaStream_t);
template cudaError_t step_launch<double>(const StepPlan&, StepArgs<double>, bool, cudaStream_t);

}  // namespace swb
