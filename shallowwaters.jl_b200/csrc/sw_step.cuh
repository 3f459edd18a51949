// sw_step.cuh -- a whole Runge-Kutta step (all stages and the dissipative
// tail) in one launch.
//
// A block owns a tile of the domain and carries it through the RKo stages of
// src/time_integration.jl:55-78 and the tail (:204-221) in shared memory: it
// loads the step's state once with a halo wide enough for every stage, keeps
// the stage input (u, v, eta) and the point-wise intermediates (q, U, V, p)
// there and writes the new state once.  Each stage is two passes over the
// tile: A forms q, U, V, p from u, v, eta (UVfluxes!, PV!, bernoulli!), B the
// tendencies and the stage combination, in place.  The tail is two more: T1
// forms the viscosity, the Laplacians and the speed, T2 the new u and v.
// Every value is formed by the expression that sw_stage.cuh and sw_tail.cuh
// form it with, so the results are theirs bit for bit.
//
// Halo.  A stage's output at (x, y) reads its input at x-2..x+1, y-2..y+1 and
// the tail reads +-2, so RKo = 4 needs 10 points below and 6 above a tile;
// halo points are computed redundantly, on rows whose number shrinks from
// stage to stage.  Walls need no extra halo: ghost points are filled in shared
// memory after each stage, by the rules of sw_ghost.cuh.  Where a periodic tile
// crosses x = 0 it holds the ghost columns of both sides: its columns run
//   ..., N-2, N-1, N, N+1 | -2, -1, 0, 1, ...
// so every column sees the neighbours and the depth that the reference's
// arrays give it, and a ghost column is 4 columns from its source.  A domain
// that fits is one tile with its ghosts.
//
// Packs.  A thread computes V columns at once (sw_pack.cuh): for Float32 a
// tile's EW lanes hold 2 EW - 4 columns, lane lx the columns lx and
// lx + EW - 4.  The two halves overlap by 4 columns; after each stage the
// lanes beside the overlap write the 3 columns that the other half cannot
// compute (it lacks their neighbours) into it.
//
// Order at the start.  What no earlier launch writes (a thread's columns and
// ghost places, the rows' static fields) is formed before the wait for the
// launch before, which it overlaps: without that 64x32 takes 1.8 us a step more,
// 512x256 1.4.  The stop flag is read beside the state.
//
// Measured (B200, us per step in blocks of steps, Smagorinsky and quadratic
// drag, the tracer of every step beside the next; the launches per stage, then
// this kernel):
//                     64x32       512x256     2048x1024   2999x1499
//   Float32        25.4    9.4  52.3  20.0    202  137    376  291
//   Float64        27.6    8.6  60.9  24.0    514  243    880  521
//   SSPRK3         35.1   13.8  46.3  25.8    338  155    641  350
//   bf16 storage   70.0   11.2  76.0  23.3    308  169    584  359
// What bounds it: the latency of its passes.  At 2048x1024 it takes 124 us alone
// for three waves of tiles; 45 % of the issue slots are used, the shared-memory
// pipe 49 %, the FMA pipe 34 %, DRAM 3 %, and a warp waits, per issue, 1.8
// cycles for the fixed latency of its packed adds, 1.2 for global loads, 0.8 each
// for barriers and shared memory (sixteen warps of 128 registers, all that the
// register file holds).  20, 24 and 32 warps with fewer registers, passes A, T1
// and T2 unrolled by 4 and a division on packs took as long or longer.  On a
// small grid a pass is one row's latency, and a step little but its ten passes.
#pragma once
#include <type_traits>

#include "sw_common.cuh"
#include "sw_ghost.cuh"
#include "sw_pack.cuh"
#include "sw_storage.cuh"

namespace swb {

constexpr int STEP_LO = 10, STEP_HI = 6;   // halo below and above a tile: 4 RK stages and the tail
constexpr int STEP_LO_SSP = 10, STEP_HI_SSP = 10;   // 4 SSP sub-stages and the tail

// How a tile reads the state, forms a stage's results and writes the new
// state.  StepNative: arrays of T.  Step16: the 16-bit storage form
// (sw_s16.cuh): pairs hi + lo scaled by s; a stage's increment b*d is rounded
// to 16 bits before it is added to the state, and so is the accumulated
// increment, which then takes the place of the accumulator X0.
struct StepNative {
    static constexpr bool S16 = false;
};
template <class E>
struct Step16 {
    static constexpr bool S16 = true;
    E* h[2][3];                         // hi of u, v, eta: the step's start, the new state
    E* l[2][3];                         // lo
    float s, inv_s;                     // scale and its inverse (powers of two)
    __device__ __forceinline__ float get(int f, int o) const { return (from16(h[0][f][o]) + from16(l[0][f][o])) * inv_s; }
    __device__ __forceinline__ void put(int f, int o, float x) const {
        const float y = x * s;
        const E hi = to16<E>(y);
        h[1][f][o] = hi;
        l[1][f][o] = to16<E>(y - from16(hi));
    }
    // the value that 16 bits keep of x
    __device__ __forceinline__ float keep(float x) const { return from16(to16<E>(x * s)) * inv_s; }
    __device__ __forceinline__ Pack<float>::P keep(Pack<float>::P x) const {
        using K = Pack<float>;
        return K::make(keep(K::get<0>(x)), keep(K::get<1>(x)));
    }
};

// Sub-stage updates (src/time_integration.jl:80-196): axb!, the kn stage's
// dxaybzc!, 4SSPRK3's caxb! and cxab!
enum StepSub : int { STEP_AXB = 0, STEP_KN = 1, STEP_4 = 2 };

template <class T>
struct StepArgs {
    Geom g;
    int ntx, nty;                       // tiles in x and y (balanced: see step_cols, step_rows)
    const T* uX; const T* vX; const T* eX;   // state at the step's start (ghosts valid)
    T* uo; T* vo; T* eo;                     // new state, with its ghosts
    SField<T> H, fq, Fx, Fy;            // fq, Fx, Fy constant along x
    using P = typename Pack<T>::P;      // constants as packs, so that they are read as they are used
    P a[4], b[4];                       // RK: RKaΔt, RKbΔt
    int stages;                         // RK stages or SSP sub-stages
    int lo, hi;                         // halo below and above a tile
    // SSP: what each sub-stage does to u1, v1, eta1 (enum StepSub) and its
    // coefficient x; kna, knb of SSPRK3's kn stage; the weights fa, fb of
    // fa*u + fb*u1 and the sub-stage after which it is taken (-1: none)
    int sub[4], combo;
    P x[4], kna, knb, fa, fb;
    T Fxt, Fyt;
    int tail, drag, smag;               // tail due; enum sw_bottom_drag; Smagorinsky (else constant νB)
    P g_, cD, rD, cSmag, nuB, Dt_diff;
    P half, q4, o12, nz;                // 1/2, 1/4, 1/12, -0.0 (sw_pack.cuh)
    GhostRule<T> gr;
    DevStatus* st;
};

// The columns of tile i: outputs [xs, xe), its first column at virtual column
// z0.  A periodic domain's first and last tile hold 4 ghost columns more, so
// the split treats the domain as 8 columns longer and gives them 4 fewer.
__host__ __device__ inline void step_cols(int N, int ep, int ntx, bool whole, int lo_, int i, int& xs, int& xe, int& z0) {
    if (whole) { xs = 0; xe = N; z0 = -2; return; }
    const int L = ep ? N + 8 : N, sh = ep ? 4 : 0;
    const int lo = (int)((long long)i * L / ntx) - sh, hi = (int)((long long)(i + 1) * L / ntx) - sh;
    xs = lo < 0 ? 0 : lo;
    xe = hi > N ? N : hi;
    z0 = xs - lo_ - (ep && i == 0 ? 4 : 0);
}
// The rows of tile j: outputs [ys, ye), loaded rows [z0, z1).
__host__ __device__ inline void step_rows(int M, int nty, int lo, int hi, int j, int& ys, int& ye, int& z0, int& z1) {
    ys = (int)((long long)j * M / nty);
    ye = (int)((long long)(j + 1) * M / nty);
    z0 = ys - lo < -2 ? -2 : ys - lo;
    z1 = ye + hi > M + 2 ? M + 2 : ye + hi;
}

// EWW warps side by side (EW = 32 EWW lanes), NW warps in all, R rows per
// thread: EH rows.
template <class T, int EWW_, int NW_, int R_>
struct StepShape {
    using P = typename Pack<T>::P;
    static constexpr int EWW = EWW_, NW = NW_, R = R_, EH = NW / EWW * R;
    static constexpr int V = Pack<T>::V, EW = 32 * EWW, NG = NW / EWW, NP = EW * EH;
    static constexpr int COLS = V == 2 ? 2 * EW - 4 : EW;     // distinct columns
    static constexpr int PAD = 4;       // the first row's left neighbour (every other read outside an array is in the next)
    static constexpr int smem(bool hvar) { return ((7 + hvar) * NP + PAD + 4 * EH) * (int)sizeof(P); }
};

// One tile.  SSP: sub-stages of the SSP schemes instead of RK stages.  SAD:
// PV_Sadourny! instead of PV_ArakawaHsu!.  EDGE is false for tiles none of
// whose points is a ghost, a ghost source or a wall.  HVAR: the depth varies along x (an array in shared
// memory; else one value per row).
template <class T, class SH, bool HVAR, bool SSP, bool SAD, bool EDGE, class IO>
__device__ __forceinline__ void step_tile(const StepArgs<T>& A, const IO& io, typename Pack<T>::P* sm, int xs, int xe, int zx,
                                          int ys, int ye, int zy, int zy1, bool whole) {
    using K = Pack<T>;
    using P = typename K::P;
    constexpr int EW = SH::EW, NP = SH::NP, R = SH::R, V = SH::V, EH = SH::EH;
    constexpr int SHIFT = EW - 4;                         // columns between the halves
    P* const su = sm + SH::PAD;
    P* const sv = su + NP;
    P* se = sv + NP;                                      // SSP: exchanged with sq after each sub-stage
    P* sq = se + NP;
    P* const sU = sv + 3 * NP;
    P* const sV = sU + NP;
    P* const sp = sV + NP;
    P* const sH = sp + NP;                                // HVAR only
    P* const tH = sH + (HVAR ? NP : 0);         // per row: depth, Coriolis, wind
    P* const tf = tH + EH;
    P* const tFx = tf + EH;
    P* const tFy = tFx + EH;

    const Geom& g = A.g;
    const int N = g.N, M = g.M;
    const bool per = g.ep != 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lx = (warp % SH::EWW) * 32 + lane;
    const int ly0 = (warp / SH::EWW) * R;
    const int EHv = zy1 - zy;                             // rows of this tile
    const P half = A.half, q4 = A.q4, nz = A.nz;
    const bool lowwall = zy == -2, highwall = zy1 == M + 2;

    // This warp's rows of [from, to) in the passes that keep nothing in
    // registers from one to the next: an equal share, as the rows shrink from
    // stage to stage and a tile's outputs are half to three quarters of its rows
    // (its own rows instead take longer: 512x256 1.9 us a step, 2048x1024 2.3,
    // SSPRK3 200x100 Float64 6.9).  With one row per thread its own, which is
    // known not to loop (64x32 1.2 us less).
    auto share = [&](int from, int to, int& r0, int& r1) {
        if constexpr (R == 1) {
            r0 = max(ly0, from);
            r1 = min(ly0 + 1, to);
        } else {
            const int n = (to - from + SH::NG - 1) / SH::NG;
            r0 = from + warp / SH::EWW * n;
            r1 = min(r0 + n, to);
        }
    };

    // this thread's columns
    int X[V];
    bool cv[V];
#pragma unroll
    for (int h = 0; h < V; h++) {
        const int z = zx + lx + h * SHIFT;
        X[h] = z;
        cv[h] = true;
        if (EDGE) {
            if (per && z < -2) X[h] = z + N + 4;
            if (per && z > N + 1) X[h] = z - (N + 4);
            cv[h] = X[h] >= -2 && X[h] <= N + 1 && !(whole && z > N + 1);
            if (!cv[h]) X[h] = 0;
        }
    }
    auto gofs = [&](int h, int y) { return (y + ROW0) * g.P + X[h] + COL0; };
    // columns whose outputs this half of the pack computes from valid neighbours
    const bool prod = V == 1 || (lx >= 2 && lx <= EW - 2);
    // the overlap: lane 3 passes its upper column down, lanes EW-4, EW-3 their lower columns up
    const bool xch = V == 2 && (lx == 3 || lx == EW - 4 || lx == EW - 3);
    const int xofs = lx == 3 ? 2 * (EW - 4) : -2 * SHIFT + 1;
    auto scalar = [](P* f) { return reinterpret_cast<T*>(f); };
    auto at = [](P* f, int s, int h) -> T& { return reinterpret_cast<T*>(f)[s * V + h]; };
    bool own[V];                                          // outputs of this tile
#pragma unroll
    for (int h = 0; h < V; h++) {
        const int rel = lx + h * SHIFT;
        own[h] = rel >= xs - zx && rel < xe - zx && (V == 1 || (h == 0 ? lx <= EW - 3 : lx >= 2));
    }

    // EDGE only: what the thread's columns are
    bool cu[V];                                           // u interior
    bool zero = false;                                    // one of the columns is 0 of a periodic domain
    bool wc[V], wrap = false;                             // a column is -1 of a periodic domain
#pragma unroll
    for (int h = 0; h < V; h++) {
        cu[h] = cv[h] && X[h] >= (per ? 0 : 1) && X[h] < N;
        zero = zero || (per && cv[h] && X[h] == 0);
        wc[h] = EDGE && per && cv[h] && X[h] == -1;
        wrap = wrap || wc[h];
    }
    P x0u[SSP ? 1 : R], x0v[SSP ? 1 : R], x0e[SSP ? 1 : R];   // RK: the accumulator X0 of this thread's points
    // RK: the step's state of this thread's points, where there are registers for it (512x256, four rows: 23.7 us a
    // step against 24.6 with a load per stage)
    constexpr bool KEEPX = !SSP && R <= 4;
    P Xku[KEEPX ? R : 1], Xkv[KEEPX ? R : 1], Xke[KEEPX ? R : 1];
    bool keep[V];                                         // nonperiodic u column that keeps its value
#pragma unroll
    for (int h = 0; h < V; h++) keep[h] = EDGE && cv[h] && !per && X[h] >= -1 && (X[h] <= 0 || X[h] >= N);
    bool ring[V];                                         // ... and is not an output column, but this tile's to write
#pragma unroll
    for (int h = 0; h < V; h++)
        ring[h] = keep[h] && !own[h] && (X[h] == -1 || X[h] >= N) && (X[h] < 0 ? xs == 0 : xe == N) &&
                  (V == 1 || (h == 0 ? lx <= EW - 3 : lx >= 2));
    // whether any lane's are
    const bool wzero = EDGE && __any_sync(0xffffffffu, zero),
               wkeep = EDGE && __any_sync(0xffffffffu, !prod && (keep[0] || keep[V - 1]));

    // stores the updated pack of index s.  Ghost points and columns outside the
    // domain receive values without meaning here: ghosts() fills the former,
    // nothing reads the latter.
    auto store = [&](P* f, int s, P val) {
        if (prod) f[s] = val;
        if (xch) scalar(f)[s * V + xofs] = lx == 3 ? K::template get<1>(val) : K::template get<0>(val);
    };
    // the same for u: its untouched columns are updated without neighbours
    auto store_u = [&](int s, P val) {
        store(su, s, val);
        if (EDGE && wkeep && !prod) {
            if (keep[0]) at(su, s, 0) = K::template get<0>(val);
            if (V == 2 && keep[V - 1]) at(su, s, V - 1) = K::template get<1>(val);
        }
    };
    // EDGE: ghost points of u, v, eta (src/ghost_points.jl:46-133), spread over
    // the block: columns -2, -1, N, N+1 of every row, then rows -2, -1, M, M+1
    // of every column; at most one of each kind per thread.  Neither kind reads
    // what the other writes.  Their places: a source, a place (with a mark
    // if the other half holds that column too), eta's source.
    constexpr int BOTH = 1 << 30;
    auto place = [&](int rel, int ly) {
        return rel < EW ? (ly * EW + rel) * V | (V == 2 && rel >= SHIFT ? BOTH : 0) : (ly * EW + rel - SHIFT) * V + V - 1;
    };
    auto source = [&](int rel, int ly) {
        return V == 1 || rel < EW - 2 ? (ly * EW + rel) * V : (ly * EW + rel - SHIFT) * V + V - 1;
    };
    auto put = [&](P* f, int at_, T val) {
        const int q = at_ & ~BOTH;
        scalar(f)[q] = val;
        if (at_ & BOTH) scalar(f)[q - SHIFT * V + V - 1] = val;
    };
    struct Places {
        int c_src = -1, c_dst = 0, c_eta = -1, c_ofs = 0;     // a column's ghost; where it is in the fields' arrays
        int r_src = -1, r_dst = 0, r_ofs = 0;                 // a row's ghost
        bool r_u = false, r_e = false;
        bool c_out = false, c_oute = false, r_outu = false, r_oute = false;   // ghosts of this tile's outputs
    };
    auto find = [&]() {
        Places G;
        static_assert(4 * EH <= SH::NW * 32 && 512 <= SH::NW * 32, "one ghost of each kind per thread");
        const int t = threadIdx.x;
        if (t < 4 * EH) {
            const int j = t & 3, ly = t >> 2, y = zy + ly;
            const bool seam = per && !whole;
            const int gx = j < 2 ? j - 2 : N + j - 2;
            const int rel = (seam ? (j < 2 ? gx : gx - (N + 4)) + (zx < -2 ? 0 : N + 4) : gx) - zx;
            const int d = per ? (whole ? (j < 2 ? N : -N) : (j < 2 ? -4 : 4)) : (j == 0 ? 3 : j == 1 ? 1 : j == 2 ? -1 : -3);
            if (ly < EHv && rel >= 0 && rel < SH::COLS && rel + d >= 0 && rel + d < SH::COLS) {
                G.c_src = source(rel + d, ly);
                G.c_dst = place(rel, ly);
                G.c_ofs = (y + ROW0) * g.P + gx + COL0;
                // eta: one ghost column each side; the corners take the column-copied value
                if ((j == 1 || j == 2) && y >= -1 && y <= M) G.c_eta = source(rel + d, min(max(ly, -zy), M - 1 - zy));
                const bool mine = rel + d >= xs - zx && rel + d < xe - zx;
                G.c_out = mine && y >= (ys == 0 ? -1 - per : ys) && y < (ye == M ? M + 2 : ye);
                G.c_oute = mine && y >= (ys == 0 ? -1 : ys) && y < (ye == M ? M + 1 : ye);
            }
        }
        if ((lowwall || highwall) && t < 512) {
            const int j = t >> 7, rel = t & 127;
            const int y = j < 2 ? j - 2 : M + j - 2, ly = y - zy;
            const int d = j == 0 ? 3 : j == 1 ? 1 : j == 2 ? -1 : -3;
            int x = zx + rel;
            if (per && x < -2) x += N + 4;
            else if (per && !whole && x > N + 1) x -= N + 4;
            if (rel < SH::COLS && ly >= 0 && ly < EHv && x >= -1 && x <= N + 1) {
                G.r_u = !per;
                G.r_e = (j == 1 || j == 2) && x >= 0 && x < N;
                if (G.r_u || G.r_e) {
                    G.r_src = source(rel, ly + d);
                    G.r_dst = place(rel, ly);
                    G.r_ofs = (y + ROW0) * g.P + x + COL0;
                    const bool in = rel >= xs - zx && rel < xe - zx, wall = j < 2 ? ys == 0 : ye == M;
                    G.r_outu = wall && (in || (x < 0 && xs == 0) || (x >= N && xe == N));
                    G.r_oute = wall && in;
                }
            }
        }
        return G;
    };
    // What the stages need of them, in one register each (found anew in each
    // stage they took 500 of a ghost pass's 900 clocks, kept as they are the
    // registers of the four-row tiles and more): source, place and its mark, and
    // what eta does (1 the same, 2 and 3 the row after or before: the corners) or
    // which of u and eta there is.
    static_assert(NP * V <= 8192, "13 bits for a place");
    int col_ghost = -1, row_ghost = -1;
    if (EDGE) {
        const Places G = find();
        const int eta = G.c_eta < 0 ? 0 : G.c_eta == G.c_src ? 1 : G.c_eta > G.c_src ? 2 : 3;
        auto packed = [](int src, int dst, int how) {
            return src < 0 ? -1 : src | (dst & ~BOTH) << 13 | (dst & BOTH ? 1 << 26 : 0) | how << 27;
        };
        col_ghost = packed(G.c_src, G.c_dst, eta);
        row_ghost = packed(G.r_src, G.r_dst, G.r_u + 2 * G.r_e);
    }

    // the rows' static fields; up to here nothing depends on the launch before
    // this one, which may still run
    for (int ly = threadIdx.x; ly < EHv; ly += SH::NW * 32) {
        const int y = zy + ly + ROW0;
        if (!HVAR) tH[ly] = K::all(A.H.p[y * A.H.sy]);
        tf[ly] = K::all(A.fq.p[y * A.fq.sy]);
        tFx[ly] = K::all(A.Fxt * A.Fx.p[y * A.Fx.sy]);
        tFy[ly] = K::all(A.Fyt * A.Fy.p[y * A.Fy.sy]);
    }
    cudaGridDependencySynchronize();
    const int stop = A.st->stop;
    // ---- the step's state, halo and ghosts included
#pragma unroll
    for (int i = 0; i < R; i++) {
        const int ly = ly0 + i;
        if (ly < EHv) {
            T a[V], b[V], c[V], d[V];
#pragma unroll
            for (int h = 0; h < V; h++) {
                a[h] = b[h] = c[h] = T(0);
                d[h] = T(1);
                if (!EDGE || cv[h]) {
                    const int o = gofs(h, zy + ly);
                    if constexpr (IO::S16) { a[h] = io.get(0, o); b[h] = io.get(1, o); c[h] = io.get(2, o); }
                    else { a[h] = A.uX[o]; b[h] = A.vX[o]; c[h] = A.eX[o]; }
                    if (HVAR) {
                        const T w = A.H.at(X[h], zy + ly);
                        d[h] = (X[h] >= -1 && X[h] <= N) ? w : T(1);
                    }
                }
            }
            const int s = ly * EW + lx;
            su[s] = K::make(a[0], a[V - 1]);
            sv[s] = K::make(b[0], b[V - 1]);
            se[s] = K::make(c[0], c[V - 1]);
            if constexpr (IO::S16) x0u[i] = x0v[i] = x0e[i] = K::all(T(0));
            else if constexpr (!SSP) { x0u[i] = su[s]; x0v[i] = sv[s]; x0e[i] = se[s]; }
            if constexpr (KEEPX) { Xku[i] = su[s]; Xkv[i] = sv[s]; Xke[i] = se[s]; }
            if (HVAR) sH[s] = K::make(d[0], d[V - 1]);
        }
    }
    if (stop) return;                                     // read beside the state
    __syncthreads();

    const T oma = A.gr.oma;
    auto ghosts = [&]() {
        auto dst = [](int p) { return (p >> 13 & 8191) | (p >> 26 & 1 ? BOTH : 0); };
        if (col_ghost >= 0) {
            const int src = col_ghost & 8191, to = dst(col_ghost), eta = col_ghost >> 27;
            if (per) put(su, to, scalar(su)[src]);
            const T w = scalar(sv)[src];
            put(sv, to, per ? w : oma * w);
            if (eta) put(se, to, scalar(se)[src + (eta == 2 ? EW * V : eta == 3 ? -EW * V : 0)]);
        }
        if (row_ghost >= 0) {
            const int src = row_ghost & 8191, to = dst(row_ghost), how = row_ghost >> 27;
            if (how & 1) put(su, to, oma * scalar(su)[src]);
            if (how & 2) put(se, to, scalar(se)[src]);
        }
    };
    auto out = [&](int f, int o, T val) {                 // a value of the new state
        if constexpr (IO::S16) io.put(f, o, val);
        else (f == 0 ? A.uo : f == 1 ? A.vo : A.eo)[o] = val;
    };

    const int stages = A.stages;
    for (int k = 0; k < stages; k++) {
        const bool last = k == stages - 1;
        // rows of the stage input that are valid, then the rows each pass forms
        const int ay = lowwall ? 0 : 2 * k, by = highwall ? EHv : EHv - (SSP ? 2 : 1) * k;
        const int a0 = lowwall ? -zy : ay + 1, a1 = highwall ? M + 1 - zy : by;
        // ---- pass A: q, U, V, p
        {
            const P gg = A.g_;
            int r0, r1;
            share(a0, a1, r0, r1);
            if (r0 < r1) {
                int s = r0 * EW + lx;
                P u_m = su[s - EW], v_c = sv[s], h_m, hs_m;
                {
                    const P Hc = HVAR ? sH[s - EW] : tH[r0 - 1];
                    h_m = K::add(se[s - EW], Hc);
                    hs_m = K::mul(q4, K::add(K::add(se[s - EW - 1], HVAR ? sH[s - EW - 1] : Hc), h_m), nz);
                }
#pragma unroll 2
                for (int ly = r0; ly < r1; ly++) {
                    const P u_c = su[s], u_r = su[s + 1], v_l = sv[s - 1], v_n = sv[s + EW], e_c = se[s];
                    const P Hc = HVAR ? sH[s] : tH[ly];
                    const P h = K::add(e_c, Hc);                        // thickness! (src/rhs.jl:131-139)
                    const P hl = K::add(se[s - 1], HVAR ? sH[s - 1] : Hc);
                    const P hlh = K::add(hl, h);
                    const P hs = K::mul(q4, hlh, nz);
                    // PV! (src/PV_advection.jl:2-18)
                    const P q = K::div(K::sub(K::add(tf[ly], K::sub(v_c, v_l)), K::sub(u_c, u_m)), K::add(hs_m, hs));
                    if (EDGE && wrap) {                     // but column -1: see below
                        if (!wc[0]) at(sq, s, 0) = K::template get<0>(q);
                        if (V == 2 && !wc[V - 1]) at(sq, s, V - 1) = K::template get<V - 1>(q);
                    } else {
                        sq[s] = q;
                    }
                    sU[s] = K::mulx(u_c, K::mulx(half, hlh));           // Uflux!/Vflux! (src/rhs.jl:277-304)
                    sV[s] = K::mulx(v_c, K::mulx(half, K::add(h, h_m)));
                    // bernoulli! (src/rhs.jl:162-180)
                    const P KEu = K::mul(half, K::add(K::mul(u_r, u_r, nz), K::mul(u_c, u_c, nz)), nz);
                    const P KEv = K::mul(half, K::add(K::mul(v_n, v_n, nz), K::mul(v_c, v_c, nz)), nz);
                    sp[s] = K::add(K::mul(half, K::add(KEu, KEv), nz), K::mul(gg, e_c, nz));
                    u_m = u_c; h_m = h; hs_m = hs; v_c = v_n;
                    s += EW;
                }
            }
        }
        if (EDGE && per) {
            // Column -1 evaluates q[end] (src/PV_advection.jl:110,126) at column N, with its own Coriolis value: a thread
            // per row (its lane held up its warp in every row: pass A of such a tile 6.2 thousand clocks instead of 4.2).
            const int rel = -1 - zx + (whole || zx < -2 ? 0 : N + 4), ly = threadIdx.x;
            if (rel >= 0 && rel < SH::COLS && ly >= a0 && ly < a1) {
                int w = rel + (whole ? N + 1 : -3), ha = 0;
                if (V == 2 && w >= EW) { w -= SHIFT; ha = V - 1; }
                w += ly * EW;
                auto hv = [&](int o, int row) { return at(se, o, ha) + (HVAR ? at(sH, o, ha) : at(tH, row, 0)); };
                const T qt = T(0.25);
                const T hq = qt * (hv(w - EW - 1, ly - 1) + hv(w - EW, ly - 1)) + qt * (hv(w - 1, ly) + hv(w, ly));
                put(sq, place(rel, ly), (at(tf, ly, 0) + (at(sv, w, ha) - at(sv, w - 1, ha)) -
                                         (at(su, w, ha) - at(su, w - EW, ha))) / hq);
            }
        }
        // X, for the next stage's input or the kn stage's snapshot, one row ahead (RK: not used on the last stage, and
        // the first row before the barrier, whose wait then hides the load: 2048x1024 134.5 -> 131.2 us a step; SSP
        // 29.2 -> 29.6, so not there)
        int o = gofs(0, zy + ly0);
        const int dX = EDGE ? X[V - 1] - X[0] : (V - 1) * SHIFT;
        P Xu = K::all(T(0)), Xv = Xu, Xe = Xu;
        auto loadX = [&]() {
            if constexpr (IO::S16) {
                Xu = K::make(io.get(0, o), io.get(0, o + dX));
                Xv = K::make(io.get(1, o), io.get(1, o + dX));
                Xe = K::make(io.get(2, o), io.get(2, o + dX));
            } else {
                Xu = K::make(A.uX[o], A.uX[o + dX]);
                Xv = K::make(A.vX[o], A.vX[o + dX]);
                Xe = K::make(A.eX[o], A.eX[o + dX]);
            }
            o += g.P;
        };
        if (!SSP && !KEEPX && ly0 < EHv) loadX();
        __syncthreads();
        // ---- pass B: tendencies and the stage combination, in place (SUB: enum StepSub, -1 for RK)
        auto pass_b = [&](auto subc) {
            constexpr int SUB = decltype(subc)::value;
            const int b0 = lowwall ? 0 : ay + 2, b1 = highwall ? EHv : by - 1;
            [[maybe_unused]] const P a = A.a[k], b = A.b[k];
            const P o12 = A.o12;
            [[maybe_unused]] const P x = A.x[k], kna = A.kna, knb = A.knb;
            if (ly0 < b1 && ly0 + R > b0) {
                int s = ly0 * EW + lx;
                P q_c = sq[s], q_l = sq[s - 1], q_r = sq[s + 1];
                P V_c = sV[s], V_l = sV[s - 1];
                P p_m = sp[s - EW];
                P qhu_part;
                if (SAD) {
                    qhu_part = K::mul(q4, K::add(sU[s - EW], sU[s - EW + 1]), nz);
                } else {
                    const P qm = sq[s - EW], qmr = sq[s - EW + 1];
                    const P qa = K::mulx(o12, K::add(K::add(qm, q_c), q_r));
                    const P qbr = K::mulx(o12, K::add(K::add(qmr, q_r), q_c));
                    qhu_part = K::add(K::mul(qa, sU[s - EW], nz), K::mul(qbr, sU[s - EW + 1], nz));
                }
                constexpr bool needX = !KEEPX && (SUB == -1 || SUB == STEP_KN);
                if (SSP && needX) loadX();
#pragma unroll (SSP ? (R < 4 ? R : 4) : R)
                for (int i = 0; i < R; i++) {
                    const int ly = ly0 + i, y = zy + ly;
                    const P Xu_ = KEEPX ? Xku[KEEPX ? i : 0] : Xu, Xv_ = KEEPX ? Xkv[KEEPX ? i : 0] : Xv;
                    [[maybe_unused]] const P Xe_ = KEEPX ? Xke[KEEPX ? i : 0] : Xe;
                    if (needX && i + 1 < R) loadX();
                    const P qn_c = sq[s + EW], qn_l = sq[s + EW - 1], qn_r = sq[s + EW + 1];
                    const P Vn_c = sV[s + EW], Vn_l = sV[s + EW - 1];
                    const P U_c = sU[s], U_r = sU[s + 1], p_c = sp[s], p_l = sp[s - 1];
                    P qhv, qhu;
                    if (SAD) {                              // PV_Sadourny! (src/PV_advection.jl:31-59)
                        qhv = K::mul(K::mulx(half, K::add(qn_c, q_c)),
                                     K::add(K::mul(q4, K::add(V_l, V_c), nz), K::mul(q4, K::add(Vn_l, Vn_c), nz)), nz);
                        const P Us = K::mul(q4, K::add(U_c, U_r), nz);
                        qhu = K::mul(K::mulx(half, K::add(q_r, q_c)), K::add(qhu_part, Us), nz);
                        qhu_part = Us;
                    } else {
                        // Arakawa-Hsu combinations (src/PV_advection.jl:88-146) at column X and, for qhu, X + 1
                        const P sc = K::add(q_c, qn_c);
                        const P qa = K::mulx(o12, K::add(sc, qn_r));
                        const P qb = K::mulx(o12, K::add(sc, qn_l));
                        P qc = K::mulx(o12, K::add(K::add(q_c, q_l), qn_c));
                        if (EDGE && wzero) {                // column 0 sums in another order
                            const P w = K::mulx(o12, K::add(sc, q_l));
                            qc = K::pick(w, qc, per && cv[0] && X[0] == 0, per && cv[V - 1] && X[V - 1] == 0);
                        }
                        const P qd = K::mulx(o12, K::add(sc, q_r));
                        const P qbr = K::mulx(o12, K::add(K::add(q_r, qn_r), qn_c));
                        const P qcr = K::mulx(o12, K::add(K::add(q_r, q_c), qn_r));
                        qhv = K::add(K::add(K::add(K::mul(qa, Vn_c, nz), K::mul(qb, Vn_l, nz)), K::mul(qc, V_l, nz)),
                                     K::mul(qd, V_c, nz));
                        qhu = K::add(K::add(qhu_part, K::mul(qcr, U_r, nz)), K::mul(qd, U_c, nz));
                        qhu_part = K::add(K::mul(qa, U_c, nz), K::mul(qbr, U_r, nz));
                    }
                    // momentum_u! (src/rhs.jl:218-245), momentum_v! (:248-274), continuity_itself! (src/continuity.jl:52-68)
                    P du = K::add(K::sub(qhv, K::sub(p_c, p_l)), tFx[ly]);
                    P dv = K::sub(tFy[ly], K::add(qhu, K::sub(p_c, p_m)));      // -(qhu + dpdy) + Fy
                    const P ds = K::add(K::sub(U_r, U_c), K::sub(Vn_c, V_c));   // -deta (RK)
                    q_c = qn_c; q_l = qn_l; q_r = qn_r; V_c = Vn_c; V_l = Vn_l; p_m = p_c;
                    if (EDGE) {
                        // untouched halo cells go through the update with a zero tendency
                        const bool row = y >= 0 && y < M;
                        du = K::pick(du, K::all(T(0)), cu[0] && row, cu[V - 1] && row);
                        if (!row || y == 0) dv = K::all(T(0));
                    }
                    if constexpr (SSP) {
                        // the momentum half of the sub-stage; eta follows from the new u, v in pass C
                        auto update = [&](P u1, P z, P d) {
                            const P xd = K::mul(x, d, nz);
                            if (SUB == STEP_AXB) return K::add(u1, xd);
                            if (SUB == STEP_KN) return K::add(K::add(K::mul(kna, u1, nz), K::mul(knb, z, nz)), xd);
                            return K::mul(half, K::add(u1, K::add(u1, xd)), nz);
                        };
                        store_u(s, update(su[s], Xu_, du));
                        store(sv, s, update(sv[s], Xv_, dv));
                    } else {
                        const P Du = K::add(x0u[i], K::mul(a, du, nz));             // axb!
                        const P Dv = K::add(x0v[i], K::mul(a, dv, nz));
                        const P De = K::sub(x0e[i], K::mul(a, ds, nz));
                        P bu = K::mul(b, du, nz), bv = K::mul(b, dv, nz), be = K::mul(b, ds, nz);
                        if constexpr (IO::S16) {
                            bu = io.keep(bu); bv = io.keep(bv); be = io.keep(be);
                            x0u[i] = io.keep(Du); x0v[i] = io.keep(Dv); x0e[i] = io.keep(De);
                        } else {
                            x0u[i] = Du; x0v[i] = Dv; x0e[i] = De;
                        }
                        P nu = K::add(Xu_, bu), nv = K::add(Xv_, bv), ne = K::sub(Xe_, be);      // caxb!
                        if (last) {
                            nu = IO::S16 ? K::add(Xu_, Du) : Du;
                            nv = IO::S16 ? K::add(Xv_, Dv) : Dv;
                            ne = IO::S16 ? K::add(Xe_, De) : De;
                        }
                        store_u(s, nu);
                        store(sv, s, nv);
                        store(se, s, ne);
                    }
                    s += EW;
                }
            }
        };
        if constexpr (!SSP) pass_b(std::integral_constant<int, -1>{});
        else if (A.sub[k] == STEP_AXB) pass_b(std::integral_constant<int, STEP_AXB>{});
        else if (A.sub[k] == STEP_KN) pass_b(std::integral_constant<int, STEP_KN>{});
        else pass_b(std::integral_constant<int, STEP_4>{});
        __syncthreads();
        if (EDGE) {
            ghosts();
            __syncthreads();
        }
        if constexpr (SSP) {
            // ---- pass C: continuity! from the new u, v and the sub-stage's eta
            // (src/continuity.jl:72-97) into sq, which takes eta's place
            const P x = A.x[k], kna = A.kna, knb = A.knb, fa = A.fa, fb = A.fb;
            const int sub = A.sub[k];
            const bool mix = k == A.combo, needX = mix || sub == STEP_KN;
            const int dX = EDGE ? X[V - 1] - X[0] : (V - 1) * SHIFT;
            int r0, r1;
            share(lowwall ? -zy : ay + 1, highwall ? M - zy : by - 1, r0, r1);
            // e at EW-2 and EW-1 of the lower half come from the upper half's lanes 2, 3
            const bool prod_e = V == 1 || (lx >= 2 && lx <= EW - 3), xch_e = V == 2 && (xch || lx == 2);
            const int xofs_e = lx <= 3 ? 2 * SHIFT : -2 * SHIFT + 1;
            if (r0 < r1) {
                int s = r0 * EW + lx;
                auto depth = [&](int o, int ly) { return K::add(se[o], HVAR ? sH[o] : tH[ly]); };
                P h_c = depth(s, r0);
                P V_c = K::mul(sv[s], K::mulx(half, K::add(h_c, depth(s - EW, r0 - 1))), nz);
#pragma unroll 2
                for (int ly = r0; ly < r1; ly++) {
                    const P h_n = depth(s + EW, ly + 1), h_l = depth(s - 1, ly), h_r = depth(s + 1, ly);
                    const P U_c = K::mul(su[s], K::mulx(half, K::add(h_c, h_l)), nz);
                    const P U_r = K::mul(su[s + 1], K::mulx(half, K::add(h_r, h_c)), nz);
                    const P V_n = K::mul(sv[s + EW], K::mulx(half, K::add(h_n, h_c)), nz);
                    const P xd = K::mul(x, K::add(K::sub(U_r, U_c), K::sub(V_n, V_c)), nz);     // -x deta
                    const P e1 = se[s];
                    P z = e1;
                    if (needX) {
                        const int o = gofs(0, zy + ly);
                        z = K::make(A.eX[o], A.eX[o + dX]);
                    }
                    P e;
                    if (sub == STEP_AXB) e = K::sub(e1, xd);
                    else if (sub == STEP_KN) e = K::sub(K::add(K::mul(kna, e1, nz), K::mul(knb, z, nz)), xd);
                    else e = K::mul(half, K::add(e1, K::sub(e1, xd)), nz);
                    if (mix) e = K::add(K::mul(fa, z, nz), K::mul(fb, e, nz));
                    if (prod_e) sq[s] = e;
                    if (xch_e) scalar(sq)[s * V + xofs_e] = lx <= 3 ? K::template get<1>(e) : K::template get<0>(e);
                    h_c = h_n; V_c = V_n;
                    s += EW;
                }
            }
            __syncthreads();
            P* const t = se; se = sq; sq = t;
            if (mix) {
                // cxayb! of u, v with the state at the step's start (:107-109, :186-191)
                for (int ly = ly0; ly < min(ly0 + R, EHv); ly++) {
                    const int s = ly * EW + lx, o = gofs(0, zy + ly);
                    su[s] = K::add(K::mul(fa, K::make(A.uX[o], A.uX[o + dX]), nz), K::mul(fb, su[s], nz));
                    sv[s] = K::add(K::mul(fa, K::make(A.vX[o], A.vX[o + dX]), nz), K::mul(fb, sv[s], nz));
                }
                __syncthreads();
            }
            if (EDGE) {
                ghosts();
                __syncthreads();
            }
        }
    }

    // ---- tail.  T1: ν (sq), Lu (sU), Lv (sV), sqrt(KE) (sp) on the tile and one point around it
    const bool quad = A.drag == SW_DRAG_QUADRATIC, smag = A.smag != 0;
    if (A.tail) {
        int r0, r1;
        share(max(ys - 1 - zy, lowwall ? 1 : 0), ye + 1 - zy, r0, r1);
        if (r0 < r1) {
            const P cS = A.cSmag;
            int s = r0 * EW + lx;
            P u_m = su[s - EW], v_m = sv[s - EW];
            P u_c = su[s], u_r = su[s + 1], v_c = sv[s], v_l = sv[s - 1], v_r = sv[s + 1];
            P DS;                                          // q4 * (DSq at corners (X, y) and (X + 1, y))
            {
                const P d = K::add(K::sub(u_c, u_m), K::sub(v_c, v_l));
                const P f = K::add(K::sub(u_r, su[s - EW + 1]), K::sub(v_r, v_c));
                DS = K::mul(q4, K::add(K::mul(d, d, nz), K::mul(f, f, nz)), nz);
            }
#pragma unroll 2
            for (int ly = r0; ly < r1; ly++) {
                const P u_n = su[s + EW], un_r = su[s + EW + 1], v_n = sv[s + EW], vn_l = sv[s + EW - 1],
                        vn_r = sv[s + EW + 1], u_l = su[s - 1];
                // ∇²! (src/gradients.jl:29-42)
                sU[s] = K::add(K::add(K::sub(u_l, u_c), K::sub(u_r, u_c)), K::add(K::sub(u_m, u_c), K::sub(u_n, u_c)));
                sV[s] = K::add(K::add(K::sub(v_l, v_c), K::sub(v_r, v_c)), K::add(K::sub(v_m, v_c), K::sub(v_n, v_c)));
                if (smag) {                                // smagorinsky_coeff! (src/diffusion.jl:68-111)
                    const P d = K::add(K::sub(u_n, u_c), K::sub(v_n, vn_l));
                    const P f = K::add(K::sub(un_r, u_r), K::sub(vn_r, v_n));
                    const P DSn = K::mul(q4, K::add(K::mul(d, d, nz), K::mul(f, f, nz)), nz);
                    const P t = K::add(K::sub(u_r, u_c), K::sub(v_n, v_c));
                    sq[s] = K::mulx(cS, K::root(K::add(K::add(DS, DSn), K::mul(t, t, nz))));
                    DS = DSn;
                }
                if (quad) {                                // bottom_drag_quadratic! (src/bottom_drag.jl:20-76)
                    const P KEu = K::mul(half, K::add(K::mul(u_r, u_r, nz), K::mul(u_c, u_c, nz)), nz);
                    const P KEv = K::mul(half, K::add(K::mul(v_n, v_n, nz), K::mul(v_c, v_c, nz)), nz);
                    sp[s] = K::root(K::add(KEu, KEv));
                }
                u_m = u_c; u_c = u_n; u_r = un_r;
                v_m = v_c; v_c = v_n; v_l = vn_l; v_r = vn_r;
                s += EW;
            }
        }
        __syncthreads();
    }
    // ---- T2: the new u, v, eta of the tile (and its untouched halo cells)
    {
        const int t0 = ys == 0 ? -2 : ys, t1 = ye == M ? M + 2 : ye;
        int r0, r1;
        share(t0 - zy, t1 - zy, r0, r1);
        if (r0 < r1) {
            const P cD = A.cD, rD = A.rD, Dt = A.Dt_diff, nuB = A.nuB;
            int s = r0 * EW + lx;
            P nq_c = nuB, nq_r = nuB, S12_c = nuB, S22_m = nuB, sK_m = nuB, h_m = nuB;
            P n_l = nuB, n_c = nuB, n_r = nuB, Lu_c = nuB, Lv_c = nuB;
            if (A.tail) {
                P n_m = nuB;
                Lu_c = sU[s];
                Lv_c = sV[s];
                if (smag) {
                    n_m = sq[s - EW];
                    n_l = sq[s - 1];
                    n_c = sq[s];
                    n_r = sq[s + 1];
                    nq_c = K::add(K::mul(q4, K::add(sq[s - EW - 1], n_m), nz), K::mul(q4, K::add(n_l, n_c), nz));
                    nq_r = K::add(K::mul(q4, K::add(n_m, sq[s - EW + 1]), nz), K::mul(q4, K::add(n_c, n_r), nz));
                }
                S22_m = K::mul(n_m, K::sub(Lv_c, sV[s - EW]), nz);
                S12_c = K::mul(nq_c, K::sub(Lu_c, sU[s - EW]), nz);
                if (quad) {
                    sK_m = sp[s - EW];
                    h_m = K::add(se[s - EW], HVAR ? sH[s - EW] : tH[max(r0 - 1, 0)]);
                }
            }
#pragma unroll 2
            for (int ly = r0; ly < r1; ly++) {
                const int y = zy + ly;
                const P u_c = su[s], v_c = sv[s];
                P nu = u_c, nv = v_c;
                if (A.tail) {
                    const P Lu_l = sU[s - 1], Lu_r = sU[s + 1], Lu_n = sU[s + EW];
                    const P Lv_l = sV[s - 1], Lv_r = sV[s + 1], Lv_n = sV[s + EW];
                    P nnl = nuB, nnc = nuB, nnr = nuB, nqn_c = nuB, nqn_r = nuB;
                    if (smag) {
                        nnl = sq[s + EW - 1]; nnc = sq[s + EW]; nnr = sq[s + EW + 1];
                        nqn_c = K::add(K::mul(q4, K::add(n_l, n_c), nz), K::mul(q4, K::add(nnl, nnc), nz));
                        nqn_r = K::add(K::mul(q4, K::add(n_c, n_r), nz), K::mul(q4, K::add(nnc, nnr), nz));
                    }
                    P Bu = K::all(T(0)), Bv = Bu;
                    if (quad) {
                        const P Hc = HVAR ? sH[s] : tH[ly];
                        const P h = K::add(se[s], Hc), hl = K::add(se[s - 1], HVAR ? sH[s - 1] : Hc);
                        const P sK = sp[s];
                        if (!EDGE || R == 1 || (y >= 0 && y < M)) {   // elsewhere u and v keep theirs, and h may be zero
                            Bu = K::div(K::mulx(K::mulx(cD, K::mulx(half, K::add(sK, sp[s - 1]))), u_c),
                                        K::mulx(half, K::add(h, hl)));
                            Bv = K::div(K::mulx(K::mulx(cD, K::mulx(half, K::add(sK, sK_m))), v_c),
                                        K::mulx(half, K::add(h, h_m)));
                        }
                        h_m = h; sK_m = sK;
                    } else if (A.drag == SW_DRAG_LINEAR) {
                        Bu = K::mul(rD, u_c, nz);
                        Bv = K::mul(rD, v_c, nz);
                    }
                    const P LLu1 = K::sub(K::mul(n_c, K::sub(Lu_r, Lu_c), nz), K::mul(n_l, K::sub(Lu_c, Lu_l), nz));
                    const P S12_n = K::mul(nqn_c, K::sub(Lu_n, Lu_c), nz);
                    const P LLu2 = K::sub(S12_n, S12_c);
                    const P LLv1 = K::sub(K::mul(nq_r, K::sub(Lv_r, Lv_c), nz), K::mul(nq_c, K::sub(Lv_c, Lv_l), nz));
                    const P S22 = K::mul(n_c, K::sub(Lv_n, Lv_c), nz);
                    const P LLv2 = K::sub(S22, S22_m);
                    nu = K::add(u_c, K::mul(Dt, K::add(K::add(Bu, LLu1), LLu2), nz));
                    nv = K::add(v_c, K::mul(Dt, K::add(K::add(Bv, LLv1), LLv2), nz));
                    S12_c = S12_n; S22_m = S22; nq_c = nqn_c; nq_r = nqn_r;
                    n_l = nnl; n_c = nnc; n_r = nnr; Lu_c = Lu_n; Lv_c = Lv_n;
                }
                const P ne = se[s];
                if (!EDGE) {
                    const int o = gofs(0, y);
                    if (own[0]) {
                        out(0, o, K::template get<0>(nu));
                        out(1, o, K::template get<0>(nv));
                        out(2, o, K::template get<0>(ne));
                    }
                    if (V == 2 && own[V - 1]) {
                        out(0, o + SHIFT, K::template get<V - 1>(nu));
                        out(1, o + SHIFT, K::template get<V - 1>(nv));
                        out(2, o + SHIFT, K::template get<V - 1>(ne));
                    }
                } else {
                    // untouched halo cells keep their value; the nonperiodic u columns among them belong to the
                    // first and the last tile
                    const bool row = y >= 0 && y < M;
                    nu = K::pick(nu, u_c, cu[0] && row, cu[V - 1] && row);
                    if (!row || y == 0) nv = v_c;
                    su[s] = nu;                            // sources of the ghost points
                    sv[s] = nv;
#pragma unroll
                    for (int h = 0; h < V; h++) {
                        const int o = gofs(h, y);
                        if (per ? own[h] : row && (own[h] || ring[h])) out(0, o, h ? K::template get<V - 1>(nu) : K::template get<0>(nu));
                        if (own[h] && y != -2) out(1, o, h ? K::template get<V - 1>(nv) : K::template get<0>(nv));
                        if (own[h] && row) out(2, o, h ? K::template get<V - 1>(ne) : K::template get<0>(ne));
                    }
                }
                s += EW;
            }
        }
    }
    if (EDGE) {
        // the outputs' ghost points
        const Places G = find();
        __syncthreads();
        if (G.c_out) {
            if (per) out(0, G.c_ofs, scalar(su)[G.c_src]);
            const T w = scalar(sv)[G.c_src];
            if (zy + (int)(threadIdx.x >> 2) >= -1) out(1, G.c_ofs, per ? w : oma * w);
        }
        if (G.c_oute && G.c_eta >= 0) out(2, G.c_ofs, scalar(se)[G.c_eta]);
        if (G.r_outu && G.r_u) out(0, G.r_ofs, oma * scalar(su)[G.r_src]);
        if (G.r_oute && G.r_e) out(2, G.r_ofs, scalar(se)[G.r_src]);
    }
}

// tile `tile` of the domain, by the calling block
template <class T, class SH, bool HVAR, bool SSP, bool SAD, class IO = StepNative>
__device__ __forceinline__ void step_block(const StepArgs<T>& A, int tile, typename SH::P* sm, const IO& io = IO()) {
    const Geom& g = A.g;
    const bool whole = A.ntx == 1 && g.N + 4 <= SH::COLS;
    int xs, xe, zx, ys, ye, zy, zy1;
    // tiles at the edges first: they take longer (a fifth), and would hold up the end of the last wave
    int i = tile % A.ntx, j = tile / A.ntx;
    if (A.ntx > 2 && A.nty > 2) {
        const int ends = 2 * A.ntx, sides = 2 * (A.nty - 2);
        if (tile < ends) {
            j = tile < A.ntx ? 0 : A.nty - 1;
        } else if (tile < ends + sides) {
            i = (tile - ends) & 1 ? A.ntx - 1 : 0;
            j = 1 + (tile - ends) / 2;
        } else {
            const int t = tile - ends - sides;
            i = 1 + t % (A.ntx - 2);
            j = 1 + t / (A.ntx - 2);
        }
    }
    step_cols(g.N, g.ep, A.ntx, whole, A.lo, i, xs, xe, zx);
    step_rows(g.M, A.nty, A.lo, A.hi, j, ys, ye, zy, zy1);
    const bool edge = zx < 2 || zx + SH::COLS > g.N - 2 || zy < 2 || zy1 > g.M - 2;
    if (edge) step_tile<T, SH, HVAR, SSP, SAD, true>(A, io, sm, xs, xe, zx, ys, ye, zy, zy1, whole);
    else step_tile<T, SH, HVAR, SSP, SAD, false>(A, io, sm, xs, xe, zx, ys, ye, zy, zy1, false);
}

template <class T, class SH, bool HVAR, bool SSP, bool SAD>
__global__ void __launch_bounds__(SH::NW * 32, 1) rk_step_kernel(const __grid_constant__ StepArgs<T> A) {
    extern __shared__ __align__(16) unsigned char step_smem[];
    // all blocks of this launch run at once on a small grid: the next launch may then be prepared
    // beside it (step_tile waits for this one's end before it reads the state)
    cudaTriggerProgrammaticLaunchCompletion();
    step_block<T, SH, HVAR, SSP, SAD>(A, (int)blockIdx.x, reinterpret_cast<typename SH::P*>(step_smem));
}

}  // namespace swb
