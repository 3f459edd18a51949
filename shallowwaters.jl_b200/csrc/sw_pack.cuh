// sw_pack.cuh -- two Float32 columns in one register pair, or one Float64.
//
// The whole-step kernel (sw_step.cuh) is written over a pack P of V columns.
// For Float32 V = 2 and the operations are the packed f32x2 instructions of
// sm_100a, each lane rounded like the scalar instruction: half the issue slots
// and half the shared-memory instructions per column.  (The FP32 pipe itself
// takes as long for a packed instruction as for two scalar ones: 128
// operations per clock and SM, measured, either way.)
//
// ptxas contracts a packed multiplication into the addition that follows it
// where both operands are products, whatever -fmad says (measured: 40 % of
// a*b + c*d differ in the last bit from the two rounded products).  A product
// that feeds a sum is therefore formed as fma(a, b, -0.0) with the -0.0 taken
// from a kernel argument: that is the rounded product exactly (signed zeros
// included), and an fma cannot be contracted further.  The fast build lets
// ptxas contract.
#pragma once
#include <cstring>

#include "sw_common.cuh"

namespace swb {

template <class T>
struct Pack;

template <>
struct Pack<float> {
    static constexpr int V = 2;
    struct P { unsigned long long v; };
    static P host(float a) {
        unsigned u;
        std::memcpy(&u, &a, 4);
        return P{(unsigned long long)u << 32 | u};
    }
    static __device__ __forceinline__ P make(float a, float b) {
        P r;
        asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
        return r;
    }
    static __device__ __forceinline__ P all(float a) { return make(a, a); }
    template <int H>
    static __device__ __forceinline__ float get(P p) {
        float a, b;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p.v));
        return H ? b : a;
    }
    static __device__ __forceinline__ P add(P a, P b) {
        P r;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
        return r;
    }
    static __device__ __forceinline__ P sub(P a, P b) {
        P r;
        asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
        return r;
    }
    // a product that feeds no sum
    static __device__ __forceinline__ P mulx(P a, P b) {
        P r;
        asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
        return r;
    }
    static __device__ __forceinline__ P mul(P a, P b, P nz) {
#if SWB_FAST_BUILD   // 0 or undefined in the parity build
        return mulx(a, b);
#else
        P r;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(nz.v));
        return r;
#endif
    }
    static __device__ __forceinline__ P div(P a, P b) { return make(get<0>(a) / get<0>(b), get<1>(a) / get<1>(b)); }
    static __device__ __forceinline__ P root(P a) { return make(sqrtf(get<0>(a)), sqrtf(get<1>(a))); }
    static __device__ __forceinline__ P pick(P a, P b, bool k0, bool k1) {   // per column: k ? a : b
        return make(k0 ? get<0>(a) : get<0>(b), k1 ? get<1>(a) : get<1>(b));
    }
};

template <>
struct Pack<double> {
    static constexpr int V = 1;
    struct P { double v; };
    static P host(double a) { return P{a}; }
    static __device__ __forceinline__ P make(double a, double) { return P{a}; }
    static __device__ __forceinline__ P all(double a) { return P{a}; }
    template <int H>
    static __device__ __forceinline__ double get(P p) { return p.v; }
    static __device__ __forceinline__ P add(P a, P b) { return P{a.v + b.v}; }
    static __device__ __forceinline__ P sub(P a, P b) { return P{a.v - b.v}; }
    static __device__ __forceinline__ P mulx(P a, P b) { return P{a.v * b.v}; }
    static __device__ __forceinline__ P mul(P a, P b, P) { return P{a.v * b.v}; }
    static __device__ __forceinline__ P div(P a, P b) { return P{a.v / b.v}; }
    static __device__ __forceinline__ P root(P a) { return P{sqrt(a.v)}; }
    static __device__ __forceinline__ P pick(P a, P b, bool k0, bool) { return k0 ? a : b; }
};

}  // namespace swb
