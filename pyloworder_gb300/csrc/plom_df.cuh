// Double-float arithmetic (an unevaluated sum hi + lo of two FP32 numbers,
// ~48 significant bits) on the FP32 pipe, and the column orderings of the
// one-sided Jacobi kernels.  GB300 runs FP64 at 1/64 of its FP32 rate, with a
// latency to match; a double-float multiply-add is 12 FP32 instructions.
// The products that are split exactly are taken with __fmul_rn: contracted into
// a later sum they would be exact there, and their rounding error, which is
// added apart, would count twice (dots of unit vectors then carry 1e-8).
#pragma once
#include <cuda_runtime.h>

namespace plom {

__device__ __forceinline__ float2 df_split(double v) {
  const float h = (float)v;
  return make_float2(h, (float)(v - (double)h));
}
__device__ __forceinline__ double df_val(float2 a) { return (double)a.x + (double)a.y; }
__device__ __forceinline__ float2 two_sum(float a, float b) {
  const float s = a + b;
  const float bb = s - a;
  return make_float2(s, (a - (s - bb)) + (b - bb));
}
__device__ __forceinline__ float2 fast_two_sum(float a, float b) {
  const float s = a + b;
  return make_float2(s, b - (s - a));
}
// a - t b
__device__ __forceinline__ float2 df_fms(float2 a, float2 t, float2 b) {
  const float ph = __fmul_rn(t.x, b.x);
  float pe = fmaf(t.x, b.x, -ph);
  pe = fmaf(t.x, b.y, pe);
  pe = fmaf(t.y, b.x, pe);
  const float2 sm = two_sum(a.x, -ph);
  return fast_two_sum(sm.x, sm.y + (a.y - pe));
}
// acc += x y (acc.y collects the low-order parts)
__device__ __forceinline__ void df_dot_acc(float2& acc, float2 x, float2 y) {
  const float ph = __fmul_rn(x.x, y.x);
  float pe = fmaf(x.x, y.x, -ph);
  pe = fmaf(x.x, y.y, pe);
  pe = fmaf(x.y, y.x, pe);
  const float2 sm = two_sum(acc.x, ph);
  acc.x = sm.x;
  acc.y += sm.y + pe;
}
__device__ __forceinline__ float2 df_mul(float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = fmaf(a.x, b.x, -p);
  e = fmaf(a.x, b.y, e);
  e = fmaf(a.y, b.x, e);
  return fast_two_sum(p, e);
}
__device__ __forceinline__ float2 df_add2(float2 a, float2 b) {
  const float2 s = two_sum(a.x, b.x);
  return fast_two_sum(s.x, s.y + (a.y + b.y));
}
__device__ __forceinline__ float2 df_mulf(float2 a, float t) {
  const float p = __fmul_rn(a.x, t);
  const float e = fmaf(a.x, t, -p);
  return fast_two_sum(p, fmaf(a.y, t, e));
}
// 1 / d in double-float
__device__ __forceinline__ float2 df_recip(float2 d) {
  const float h = __fdividef(1.0f, d.x);
  const float r = fmaf(-d.x, h, 1.0f) - d.y * h;
  return fast_two_sum(h, r * h);
}
// d^-1/2 in double-float (d > 0): an FP32 estimate and one Newton step
__device__ __forceinline__ float2 df_rsqrt(float2 d) {
  const float y0 = rsqrtf(d.x);
  const float q = __fmul_rn(y0, y0), qe = fmaf(y0, y0, -q);
  const float r = fmaf(-d.x, q, 1.0f) - fmaf(d.x, qe, d.y * q);
  return fast_two_sum(y0, 0.5f * y0 * r);
}

// round-robin (circle method) over np (even) players; np - 1 steps
__device__ __forceinline__ void rr_pair(int step, int k, int np, int& a, int& b) {
  const int m = np - 1;
  if (k == 0) {
    a = 0;
    b = 1 + (step % m);
  } else {
    a = 1 + (step + k) % m;
    b = 1 + (step - k + m) % m;
  }
}
// rounds of the 6 pairs inside a block of 4: (0,1)(2,3) / (0,2)(1,3) / (0,3)(1,2)
__device__ __forceinline__ void intra_pair(int round, int which, int& a, int& b) {
  if (which == 0) {
    a = 0;
    b = round + 1;
  } else {
    a = (round == 0) ? 2 : 1;
    b = (round == 2) ? 2 : 3;
  }
}

}  // namespace plom
