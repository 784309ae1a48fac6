// twofloat.cuh -- sums in pairs of FP32 numbers (hi + lo), for the reductions
// whose FP32 results need more than FP32 sums.  GB300 does about 1.2 FP64
// TFLOP/s against 80 in FP32, so a pair of floats per sum (Knuth's two-sum,
// Dekker / Ogita-Rump-Oishi cascaded summation: error about n 2^-48 sum |x|)
// replaces an FP64 accumulator where it would bound the kernel.
#pragma once

#include "ptx.cuh"

namespace msot {

// s + c carries the sum; two instances (or frames) side by side
struct Sum2 {
    float2 s, c;
    __device__ __forceinline__ void zero() { s = c = make_float2(0.f, 0.f); }
    // adds x and the small correction e (an exact product's tail, or zero)
    __device__ __forceinline__ void add(float2 x, float2 e) {
        const float2 m1 = make_float2(-1.f, -1.f);
        const float2 t = fadd2(s, x);
        const float2 bb = ffma2(s, m1, t);               // t - s
        const float2 ea = ffma2(ffma2(bb, m1, t), m1, s);  // s - (t - bb)
        const float2 eb = ffma2(bb, m1, x);              // x - bb
        s = t;
        c = fadd2(c, fadd2(e, fadd2(ea, eb)));
    }
    __device__ __forceinline__ void add(float2 x) {
        const float2 m1 = make_float2(-1.f, -1.f);
        const float2 t = fadd2(s, x);
        const float2 bb = ffma2(s, m1, t);
        const float2 ea = ffma2(ffma2(bb, m1, t), m1, s);
        const float2 eb = ffma2(bb, m1, x);
        s = t;
        c = fadd2(c, fadd2(ea, eb));
    }
    __device__ __forceinline__ double x() const { return (double)s.x + (double)c.x; }
    __device__ __forceinline__ double y() const { return (double)s.y + (double)c.y; }
};

// the scalar form
struct Sum1 {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(float x) {
        const float t = __fadd_rn(s, x);
        const float bb = __fsub_rn(t, s);
        c = __fadd_rn(c, __fadd_rn(__fsub_rn(s, __fsub_rn(t, bb)), __fsub_rn(x, bb)));
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s + (double)c; }
};

}  // namespace msot
