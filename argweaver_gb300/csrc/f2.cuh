// FP32 pair arithmetic (value = hi + lo, |lo| <= ulp(hi) / 2) for the dominant path of the
// FP32 forward and backward steps. Within a tree the normalised column converges to the
// fixed point of the step; a rounding error of the step shifts that fixed point by about the
// error divided by (1 - the chain's contraction), and with stay probabilities near 1 the
// contraction is slow. The stay, emission and rescaling factors, which carry almost all of
// a state's mass from column to column, therefore run on pairs built from error-free
// transforms (Fast2Sum, and products split by FMA); the mass moving in from other states
// (a few percent) stays plain FP32.
#pragma once

namespace awg {

struct F2 {
    float hi, lo;
};
__device__ __forceinline__ F2 f2_renorm(float a, float b) {  // |a| >= |b|
    const float s = a + b;
    return F2{s, b - (s - a)};
}
// (x.hi + x.lo) * (1 - r), 0 <= r < 1 (x.lo * r dropped: below the pair's precision)
__device__ __forceinline__ F2 f2_keep(F2 x, float r) {
    const float t = x.hi * r;
    const float h = x.hi - t;
    return f2_renorm(h, ((x.hi - h) - t) + x.lo);
}
// x * e
__device__ __forceinline__ F2 f2_mul(F2 x, float e) {
    const float p = x.hi * e;
    return f2_renorm(p, fmaf(x.hi, e, -p) + x.lo * e);
}
// a deterministic switch move (BatchDev::determprob): 1 - mv kept, or -mv where the sign is set
__device__ __forceinline__ F2 f2_move(F2 x, float mv) {
    return __float_as_int(mv) < 0 ? f2_mul(x, -mv) : f2_keep(x, mv);
}
// x + s (any magnitudes: two-sum)
__device__ __forceinline__ F2 f2_add(F2 x, float s) {
    const float h = x.hi + s;
    const float bb = h - x.hi;
    const float err = (x.hi - (h - bb)) + (s - bb);
    return f2_renorm(h, err + x.lo);
}
// x + y, both pairs
__device__ __forceinline__ F2 f2_add2(F2 x, F2 y) {
    const F2 s = f2_add(x, y.hi);
    return f2_renorm(s.hi, s.lo + y.lo);
}

}  // namespace awg
