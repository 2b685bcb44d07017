// hmf_f32x2.cuh -- two float32 values in one 64-bit register pair and the
// packed arithmetic of sm_100 and later: each operation rounds both halves to
// nearest even, denormals kept, exactly as the scalar operation does, so code
// written with it gives the scalar code's bits at half the issued
// instructions.  There is no operator*: the assembler contracts a packed
// multiplication whose only use is a packed addition into one fused operation
// (with explicit rounding and --fmad=false too: 24 % of random a * b + c
// differed from the two scalar operations), so f2_mul is a fused operation
// already, with a -0 addend that the caller takes from a kernel parameter
// (a constant would be folded): a * b + (-0) rounds to a * b, signs of zero
// included.
#pragma once

namespace hmf {

struct F2 {
  unsigned long long v;
};

__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ F2 f2(float both) { return f2(both, both); }
__device__ __forceinline__ float f2_lo(F2 a) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
  (void)hi;
  return lo;
}
__device__ __forceinline__ float f2_hi(F2 a) {
  float lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v));
  (void)lo;
  return hi;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
// a * b; neg_zero holds -0 in both halves and is not known at compile time
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b, F2 neg_zero) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(neg_zero.v));
  return r;
}
// RN(a * b + c), one rounding
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
// 8-byte aligned loads and stores of two neighbouring floats
__device__ __forceinline__ F2 f2_ld(const float* p) { return F2{*reinterpret_cast<const unsigned long long*>(p)}; }
__device__ __forceinline__ void f2_st(float* p, F2 a) { *reinterpret_cast<unsigned long long*>(p) = a.v; }
// (keep_lo ? a.lo : 0, keep_hi ? a.hi : 0)
__device__ __forceinline__ F2 f2_mask(F2 a, bool keep_lo, bool keep_hi) {
  return f2(keep_lo ? f2_lo(a) : 0.0f, keep_hi ? f2_hi(a) : 0.0f);
}
// minimum that is NaN when either operand is
__device__ __forceinline__ float min_nan(float a, float b) {
  float r;
  asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

}  // namespace hmf
