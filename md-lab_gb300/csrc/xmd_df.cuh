// xmd_df.cuh -- double-float arithmetic: a number as an unevaluated sum of
// two FP32 values (about 48 significant bits) on the FP32 pipe, which on
// GB300 issues 58 times as many operations a second as the FP64 pipe.
//
// The error-free transforms are Dekker's and Knuth's (T. J. Dekker, Numer.
// Math. 18, 1971; D. E. Knuth, TAOCP vol. 2, 4.2.2): they rely on each
// operation being rounded by itself, so they are written with the _rn
// intrinsics, which the compiler does not contract or reorder.
#pragma once

namespace xk {

struct df {
  float h, l;
};

// a + b = s + e exactly
__device__ __forceinline__ df two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
// the same for |a| >= |b| (or a = 0)
__device__ __forceinline__ df fast_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
// a b = p + e exactly
__device__ __forceinline__ df two_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}
// a + b; the low parts' sum is rounded to FP32 (2^-48 of the result unless
// the high parts cancel)
__device__ __forceinline__ df df_add(df a, df b) {
  const df s = two_sum(a.h, b.h);
  return {s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ df df_add_fast(df a, df b) {  // |a| >= |b|
  const df s = fast_two_sum(a.h, b.h);
  return {s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l))};
}
__device__ __forceinline__ df df_sub(df a, df b) { return df_add(a, {-b.h, -b.l}); }
__device__ __forceinline__ df df_mul(df a, df b) {
  const df p = two_prod(a.h, b.h);
  return {p.h, __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, p.l))};
}
// the pair with |l| at most half an ulp of h
__device__ __forceinline__ df df_norm(df a) { return fast_two_sum(a.h, a.l); }
__device__ __forceinline__ double df_value(df a) { return (double)a.h + (double)a.l; }
// c as an FP32 pair (host)
inline df df_split(double c) {
  const float h = (float)c;
  return {h, (float)(c - (double)h)};
}

}  // namespace xk
