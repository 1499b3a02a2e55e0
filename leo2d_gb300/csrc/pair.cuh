// pair.cuh - sums and products as unevaluated pairs of FP32 numbers (device code).
//
// Knuth's exact addition and the FMA's exact product: about 48 bits at FP32 cost, where
// GB300's FP64 unit takes a warp instruction every 16 cycles of an SM.
#pragma once

namespace leo2d {

// h + l, |l| at most half an ulp of h (about 2^-45 relative).
struct FPair {
  float h, l;
};
__device__ __forceinline__ FPair fpair_mul(FPair a, FPair b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  return {p, __fmaf_rn(a.l, b.h, e)};
}
__device__ __forceinline__ FPair fpair_two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), t = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, t)), __fsub_rn(b, t))};
}
__device__ __forceinline__ FPair fpair_fast_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
// a + b rounded to FP32
__device__ __forceinline__ float fpair_sum(FPair a, FPair b) {
  const FPair s = fpair_two_sum(a.h, b.h);
  return __fadd_rn(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ FPair fpair_neg(FPair a) { return {-a.h, -a.l}; }

// A running sum of FP32 terms as an unevaluated pair hi + lo: Knuth's exact
// addition (hi + x = s + e without rounding), e goes into lo. It keeps some 48 bits
// where FP64 keeps 53, at FP32 cost: GB300's FP64 unit takes a warp's addition
// every 16 cycles of an SM and answers late, so FP64 sums at the end of a step
// (a chain over the warps) were microseconds of each step. Sums over CTAs are FP64.
struct PairSum {
  float h = 0.f, l = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float s = __fadd_rn(h, x), b = __fsub_rn(s, h);
    l = __fadd_rn(l, __fadd_rn(__fsub_rn(h, __fsub_rn(s, b)), __fsub_rn(x, b)));
    h = s;
  }
  __device__ __forceinline__ void add(FPair x) {
    const FPair s = fpair_two_sum(h, x.h);
    l = __fadd_rn(l, __fadd_rn(x.l, s.l));
    h = s.h;
  }
  __device__ __forceinline__ void add(const PairSum& o) {
    add(o.h);
    l = __fadd_rn(l, o.l);
  }
  __device__ __forceinline__ PairSum shfl_xor(int o) const {
    PairSum r;
    r.h = __shfl_xor_sync(0xffffffffu, h, o);
    r.l = __shfl_xor_sync(0xffffffffu, l, o);
    return r;
  }
  // (an infinite term leaves h infinite and l undefined: the sum is infinite, as in FP64)
  __device__ __forceinline__ double value() const { return isfinite(h) ? (double)h + (double)l : (double)h; }
};

}  // namespace leo2d
