// sw_step_batch.cu -- the whole-step kernel over the tiles of an ensemble.
//
// The members' arguments travel as kernel parameters: a block reads those of
// its member from the constant bank as the lone kernel does, with an index the
// whole block shares (from device memory they would take registers that the
// kernel does not have).  Members differ in depth profile, so the depth is an
// array in shared memory for all of them.
#include <algorithm>

#include "sw_step_launch.cuh"

namespace swb {
namespace {

template <class SH>
__global__ void __launch_bounds__(SH::NW * 32, 1) rk_step_batch(const __grid_constant__ StepBatch B) {
    extern __shared__ __align__(16) unsigned char step_smem[];
    int lo = 0, hi = B.n - 1;                     // the member of this block
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (B.block0[mid] <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    if (*B.istep > B.nt[lo]) return;
    const StepArgs<float>& A = B.m[lo];
    step_block<float, SH, true, false, false>(A, (int)blockIdx.x - B.block0[lo],
                                              reinterpret_cast<typename SH::P*>(step_smem));
}

template <class SH>
cudaError_t go_batch(const StepBatch* b, int nblocks, cudaStream_t stream) {
    constexpr int smem = SH::smem(true);
    if (!b) return cudaFuncSetAttribute(rk_step_batch<SH>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    rk_step_batch<SH><<<nblocks, SH::NW * 32, smem, stream>>>(*b);
    return cudaGetLastError();
}

cudaError_t go_batch_shape(int shape, const StepBatch* b, int nblocks, cudaStream_t stream) {
    using SS = Shapes<float, true>;
    if (shape == 0) return go_batch<SS::S0>(b, nblocks, stream);
    if (shape == 1) return go_batch<SS::S1>(b, nblocks, stream);
    if (shape == 2) return go_batch<SS::S2>(b, nblocks, stream);
    if (shape == 3) return go_batch<SS::S3>(b, nblocks, stream);
    return go_batch<SS::S4>(b, nblocks, stream);
}

// a member's tiles in shape s with at most h rows each; false if it has none
bool member_tiles(const ShapeInfo& f, const Geom& g, int h, int& ntx, int& nty, double& clocks) {
    ntx = split_cols(g.N, g.ep, f.cols, STEP_LO, STEP_HI);
    if (!ntx) return false;
    const int most = g.M + 4 <= f.EH ? g.M : f.EH - STEP_LO - STEP_HI;
    nty = (g.M + std::min(h, most) - 1) / std::min(h, most);
    while (nty > 1 && g.M / nty < 2) nty--;
    const int rows = (g.M + nty - 1) / nty;
    if (rows > most) return false;
    clocks = tile_clocks(f, std::min(rows + STEP_LO + STEP_HI, g.M + 4));
    return true;
}

}  // namespace

int step_batch_plan(const Geom* gs, int n, int nsm, StepPlan* plans) {
    const auto info = shape_infos<float, true>();
    // force a shape and the most rows per tile, as for a lone context (plan_of)
    const char* env = getenv("SWB200_STEP");
    const char* envr = getenv("SWB200_STEP_ROWS");
    const int only = env ? atoi(env) : NSHAPES, rows = envr ? atoi(envr) : 0;
    int best = -1, best_h = 0;
    double cost = 1e30;
    for (int s = 0; s < NSHAPES; s++) {
        if (only < NSHAPES && s != only) continue;
        for (int h = rows > 0 ? std::max(rows, 2) : info[s].EH; h >= 2; h -= rows > 0 ? h : h > 16 ? 4 : 2) {
            double total = 0, longest = 0;
            bool ok = true;
            for (int m = 0; m < n && ok; m++) {
                int ntx, nty;
                double c;
                ok = member_tiles(info[s], gs[m], h, ntx, nty, c);
                total += ok ? ntx * nty * c : 0;
                longest = std::max(longest, ok ? c : 0);
            }
            // the blocks' clocks over the SMs, and on average half a block that the others wait for
            const double c = total / nsm + 0.5 * longest;
            if (ok && c < cost) { cost = c; best = s; best_h = h; }
        }
    }
    for (int m = 0; m < n && best >= 0; m++) {
        double c;
        plans[m].shape = best;
        member_tiles(info[best], gs[m], best_h, plans[m].ntx, plans[m].nty, c);
    }
    return best;
}

cudaError_t step_batch_prepare(int shape) { return go_batch_shape(shape, nullptr, 0, nullptr); }

cudaError_t step_batch_launch(int shape, StepBatch& b, cudaStream_t stream) {
    b.block0[0] = 0;
    for (int m = 0; m < b.n; m++) {
        set_constants<float, false>(b.m[m]);
        b.block0[m + 1] = b.block0[m] + b.m[m].ntx * b.m[m].nty;
    }
    return go_batch_shape(shape, &b, b.block0[b.n], stream);
}

}  // namespace swb
