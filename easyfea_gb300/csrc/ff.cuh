// Float-float arithmetic: a value is an unevaluated pair hi + lo of floats
// (~2^-44 relative), products by the exact FMA split, sums by TwoSum (Knuth).
// GB300 runs FP32 at 64x its FP64 rate, so work on pairs costs less than in
// FP64 even at ~12 FP32 operations each.
#pragma once

#include <cuda_runtime.h>

namespace gfea {

__device__ __forceinline__ void ff_split(double d, float& hi, float& lo) {
  hi = (float)d;
  lo = (float)(d - (double)hi);
}

__device__ __forceinline__ float2 ff_pair(double d) {
  float2 v;
  ff_split(d, v.x, v.y);
  return v;
}

// (sh, sl) += (ah, al) (bh, bl); the al bl term is below the pair's precision
__device__ __forceinline__ void ff_fma_acc(float& sh, float& sl, float ah, float al, float bh, float bl) {
  const float p = ah * bh;
  const float e = fmaf(ah, bh, -p) + fmaf(ah, bl, al * bh);
  const float t = sh + p;
  const float bp = t - sh;
  sl += ((sh - (t - bp)) + (p - bp)) + e;
  sh = t;
}

// (ah, al) - (sh, sl), normalised
__device__ __forceinline__ void ff_sub(float ah, float al, float sh, float sl, float& hi, float& lo) {
  const float t = ah - sh;
  const float bp = t - ah;
  const float err = (ah - (t - bp)) + (-sh - bp);
  const float l = err + (al - sl);
  hi = t + l;
  lo = l - (hi - t);
}

// (ah, al) (bh, bl), normalised
__device__ __forceinline__ float2 ff_mul(float2 a, float2 b) {
  const float p = a.x * b.x;
  const float e = fmaf(a.x, b.x, -p) + fmaf(a.x, b.y, a.y * b.x);
  const float h = p + e;
  return make_float2(h, e - (h - p));
}

// 1 / (ah, al): a float quotient and one correction by its exact remainder
__device__ __forceinline__ float2 ff_recip(float2 a) {
  const float r = 1.0f / a.x;
  const float c = r * (fmaf(-a.x, r, 1.0f) - a.y * r);
  const float h = r + c;
  return make_float2(h, c - (h - r));
}

}  // namespace gfea
