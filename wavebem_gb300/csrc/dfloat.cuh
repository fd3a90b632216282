// Sums and products of double-float pairs that are left unnormalised, written
// with rounded operations so that none is contracted, and conversions between them and FP64 that leave the FP64
// pipe alone: on this GPU it runs at 1/64 of the FP32 rate, and conversions
// to and from 64 bits go through it. Unnormalised: |lo| may reach a few units
// in the last place of hi.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include "common.cuh"

namespace wbem {

__device__ __forceinline__ df pair_load(float2 v) { return {v.x, v.y}; }

__device__ __forceinline__ df pair_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}

// |a| >= |b| or a = 0
__device__ __forceinline__ df pair_fast(float a, float b) {
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}

__device__ __forceinline__ df pair_prod(float a, float b) {
  const float p = __fmul_rn(a, b);
  return {p, __fmaf_rn(a, b, -p)};
}

__device__ __forceinline__ df pair_mul(df a, df b) {
  df p = pair_prod(a.hi, b.hi);
  p.lo = __fmaf_rn(a.lo, b.hi, __fmaf_rn(a.hi, b.lo, p.lo));
  return p;
}

__device__ __forceinline__ df pair_add(df a, df b) {
  df s = pair_sum(a.hi, b.hi);
  s.lo = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  return s;
}

__device__ __forceinline__ df pair_neg(df a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ df pair_sub(df a, df b) { return pair_add(a, pair_neg(b)); }
__device__ __forceinline__ df pair_norm(df a) { return pair_fast(a.hi, a.lo); }
__device__ __forceinline__ df pair_half(df a) { return {0.5f * a.hi, 0.5f * a.lo}; }

// the leading 24 bits of x, cut off; |x| < 2^127, zero below 2^-126
__device__ __forceinline__ float cut_to_float(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mag = hi & 0x7fffffffu;
  const uint32_t f = (mag - 0x38000000u) << 3 | lo >> 29;
  return mag < 0x38100000u ? 0.f : __uint_as_float(f | (hi & 0x80000000u));
}

// x as a pair: the leading 24 bits and the 29 below them (rounded to 24).
// |x| < 2^127; the lower part is left out below 2^-74.
__device__ __forceinline__ df pair_split(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t mag = hi & 0x7fffffffu;
  const float h = cut_to_float(x);
  // 2^(exponent - 52) with the sign of x
  const uint32_t e = ((mag - 0x38000000u - (52u << 20)) << 3 & 0x7f800000u) | (hi & 0x80000000u);
  const float l = __fmul_rn(__uint2float_rn(lo & 0x1fffffffu), __uint_as_float(e));
  return {h, mag < 0x3b500000u ? 0.f : l};
}

// x in 64 bits (exact; zero and values below 2^-126 give a value below 2^-125)
__device__ __forceinline__ double widen(float x) {
  const uint32_t u = __float_as_uint(x);
  return __hiloint2double((int)(((u & 0x7fffffffu) >> 3) + 0x38000000u | (u & 0x80000000u)),
                          (int)(u << 29));
}

}  // namespace wbem
