// hmf_ff.cuh -- float-float arithmetic on the FP32 pipes: a number is the
// unevaluated sum h + l of two floats, |l| <= ulp(h)/2 (about 48 bits).  This
// part's FP64 rate is 1/64 of its FP32 rate, so a result that is rounded to
// float in the end is cheaper computed this way and, where its error bound
// does not settle the rounding, once more in double.
//
// Sums and products: Dekker, "A floating-point technique for extending the
// available precision" (1971), and Joldes, Muller, Popescu, "Tight and
// rigorous error bounds for basic building blocks of double-word arithmetic"
// (ACM TOMS 44, 2017), algorithms 6 (relative error below 3.1 * 2^-48, also
// under cancellation) and 12 (below 5 * 2^-48).  Valid while nothing under- or
// overflows; the callers check their operands' ranges.
#pragma once

namespace hmf {

struct FFloat {
  float h, l;
};

__device__ __forceinline__ FFloat ff_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FFloat ff_fast_sum(float a, float b) {  // |a| >= |b| or a == 0
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FFloat ff_sum(FFloat a, FFloat b) {
  const FFloat s = ff_two_sum(a.h, b.h), t = ff_two_sum(a.l, b.l);
  const FFloat v = ff_fast_sum(s.h, __fadd_rn(s.l, t.h));
  return ff_fast_sum(v.h, __fadd_rn(t.l, v.l));
}
__device__ __forceinline__ FFloat ff_sum(FFloat a, float b) {
  const FFloat s = ff_two_sum(a.h, b);
  return ff_fast_sum(s.h, __fadd_rn(a.l, s.l));
}
__device__ __forceinline__ FFloat ff_mul(FFloat a, FFloat b) {
  const float p = __fmul_rn(a.h, b.h);
  const float e = __fmaf_rn(a.h, b.h, -p);
  const float c = __fmaf_rn(a.h, b.l, __fmaf_rn(a.l, b.h, __fmul_rn(a.l, b.l)));
  return ff_fast_sum(p, __fadd_rn(e, c));
}
__device__ __forceinline__ FFloat ff_mul(FFloat a, float b) {
  const float p = __fmul_rn(a.h, b);
  return ff_fast_sum(p, __fmaf_rn(a.l, b, __fmaf_rn(a.h, b, -p)));
}

// Whether every number within a relative `rel` of v rounds to the same float,
// which is then `out` (v.h normal and in range).
__device__ __forceinline__ bool ff_rounds(FFloat v, float rel, float& out) {
  const float e = __fmul_rn(fabsf(v.h), rel);
  out = __fadd_rn(v.h, v.l);
  return __fadd_rn(v.h, __fadd_rn(v.l, e)) == out && __fadd_rn(v.h, __fsub_rn(v.l, e)) == out;
}

// Float-float running sum (hi + lo): each term is added with Knuth's
// TwoSum, its rounding error collected in lo.  FP32 instructions only (the
// FP64 rate of this part is a small fraction of FP32's); relative error about
// n * 2^-48 after n terms of one sign, against 2^-24 for a plain float sum.
struct FF {
  float hi, lo;
};

__device__ __forceinline__ void ff_add(FF& a, float t) {
  const float s = a.hi + t;
  const float bb = s - a.hi;
  const float err = (a.hi - (s - bb)) + (t - bb);
  a.hi = s;
  a.lo += err;
}

__device__ __forceinline__ FF ff_merge(FF a, FF b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float err = (a.hi - (s - bb)) + (b.hi - bb);
  return {s, (a.lo + b.lo) + err};
}

}  // namespace hmf
