// Double-float arithmetic (device).
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace awg {
namespace {

// the built-in overloads stay visible beside the double-float ones
using ::fma;
using ::fmax;
using ::__shfl_xor_sync;

// Double-float: value = hi + lo, |lo| <= ulp(hi) / 2, about 48 significant bits, from
// FP32 error-free transforms (Knuth's two-sum; the product's error by fused multiply-add).
// The FP32 path's variant-column emissions are formed in it: the forward posterior amplifies
// an error of those emissions thousands-fold on the columns where they differ little between
// states, so they must reach FP32 as correctly rounded ratios to the column's largest. FP32
// forms left the posterior up to 6.6e-5 from FP64's (9.1e-5 with only the partials in
// double-float); double-float, 3.1e-6 (k = 64, 100,000 columns).
struct df {
    float hi, lo;
    __device__ __forceinline__ df() : hi(0.f), lo(0.f) {}
    __device__ __forceinline__ df(double x) : hi((float)x), lo((float)(x - (double)(float)x)) {}
    // small integer constants (0, 1, 4 in the emission forms) without the FP64 split
    __device__ __forceinline__ df(int x) : hi((float)x), lo(0.0f) {}
    __device__ __forceinline__ df(float h, float l) : hi(h), lo(l) {}
    __device__ __forceinline__ explicit operator double() const { return (double)hi + (double)lo; }
};
__device__ __forceinline__ df df_fast2(float a, float b) {  // |a| >= |b|
    const float s = __fadd_rn(a, b);
    return df(s, __fsub_rn(b, __fsub_rn(s, a)));
}
__device__ __forceinline__ df operator+(df a, df b) {
    const float s = __fadd_rn(a.hi, b.hi);
    const float bb = __fsub_rn(s, a.hi);
    const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bb)), __fsub_rn(b.hi, bb));
    return df_fast2(s, __fadd_rn(e, __fadd_rn(a.lo, b.lo)));
}
__device__ __forceinline__ df operator-(df a) { return df(-a.hi, -a.lo); }
__device__ __forceinline__ df operator-(df a, df b) { return a + (-b); }
__device__ __forceinline__ df operator*(df a, df b) {
    const float p = __fmul_rn(a.hi, b.hi);
    const float e = __fmaf_rn(a.hi, b.hi, -p);
    return df_fast2(p, __fmaf_rn(a.hi, b.lo, __fmaf_rn(a.lo, b.hi, e)));
}
__device__ __forceinline__ df &operator+=(df &a, df b) { return a = a + b; }
__device__ __forceinline__ bool operator<(df a, df b) { return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
// a + b for a, b >= 0 (every sum of the emission passes: partials, branch probabilities and
// their products): the larger high part first makes Dekker's fast two-sum exact, three adds
// where the two-sum of arbitrary signs takes six
__device__ __forceinline__ df df_addp(df a, df b) {
    const float big = fmaxf(a.hi, b.hi), small = fminf(a.hi, b.hi);
    const float s = __fadd_rn(big, small);
    const float e = __fsub_rn(small, __fsub_rn(s, big));
    return df_fast2(s, __fadd_rn(e, __fadd_rn(a.lo, b.lo)));
}
// a * b + c, a, b, c >= 0 (the JC69 steps of the emission passes)
__device__ __forceinline__ df fma(df a, df b, df c) { return df_addp(a * b, c); }
__device__ __forceinline__ df fmax(df a, df b) { return a < b ? b : a; }
__device__ __forceinline__ df __shfl_xor_sync(unsigned mask, df v, int o) {
    return df(::__shfl_xor_sync(mask, v.hi, o), ::__shfl_xor_sync(mask, v.lo, o));
}

}  // namespace
}  // namespace awg
