// Arithmetic of the radix-8 Stockham FFTs (fft_pass.cuh): butterflies on two
// columns at once, and the radices of a length.  Lengths N = 8^a * {1, 2, 4}
// (32 .. 4096) use radix-8 stages and at most one radix-2 or radix-4 stage; the
// output is in natural order (Stockham).
//
// Stage with radix R, p = product of the previous radices: butterfly
// i in [0, N/R) with k = i mod p reads x[i + r N/R] (r < R), multiplies by
// exp(-2 pi i r k / (p R)), takes the R-point DFT and writes it to
// y[(i - k) R + k + r p].  Forward transform: exp(-2 pi i j k / N), as cuFFT
// and numpy.
#pragma once

#include <cuda_runtime.h>

namespace gbp {
namespace fft {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmi(float2 a) { return make_float2(a.y, -a.x); }  // a * (-i)

// Two columns side by side: re = (re of column 0, re of column 1), im alike.
// One f32x2 instruction does both columns' addition, with the rounding of two
// scalar ones, and a multiplication by -i is a renaming.
struct Pair {
  float2 re, im;
};
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ Pair cadd(const Pair& a, const Pair& b) { return {add2(a.re, b.re), add2(a.im, b.im)}; }
__device__ __forceinline__ Pair csub(const Pair& a, const Pair& b) { return {sub2(a.re, b.re), sub2(a.im, b.im)}; }
__device__ __forceinline__ Pair cmi(const Pair& a) { return {a.im, make_float2(-a.re.x, -a.re.y)}; }
__device__ __forceinline__ Pair csub_mi(const Pair& a, const Pair& b) { return {sub2(a.im, b.im), sub2(b.re, a.re)}; }
__device__ __forceinline__ Pair cmul(const Pair& a, float2 w) {
  return {make_float2(a.re.x * w.x - a.im.x * w.y, a.re.y * w.x - a.im.y * w.y),
          make_float2(a.re.x * w.y + a.im.x * w.x, a.re.y * w.y + a.im.y * w.x)};
}

__device__ __forceinline__ void dft2(Pair& a, Pair& b) {
  const Pair t = a;
  a = cadd(t, b);
  b = csub(t, b);
}

__device__ __forceinline__ void dft4(Pair* u) {
  const Pair a0 = cadd(u[0], u[2]), a1 = csub(u[0], u[2]);
  const Pair a2 = cadd(u[1], u[3]), a3 = csub_mi(u[1], u[3]);
  u[0] = cadd(a0, a2);
  u[2] = csub(a0, a2);
  u[1] = cadd(a1, a3);
  u[3] = csub(a1, a3);
}

__device__ __forceinline__ void dft8(Pair* u) {
  const float r = 0.70710678118654752440f;
  const float2 s = make_float2(r, r), ns = make_float2(-r, -r);
  const Pair a0 = cadd(u[0], u[4]), a1 = csub(u[0], u[4]);
  const Pair a2 = cadd(u[2], u[6]), a3 = csub_mi(u[2], u[6]);
  const Pair a4 = cadd(u[1], u[5]), a5 = csub(u[1], u[5]);
  const Pair a6 = cadd(u[3], u[7]), a7 = csub_mi(u[3], u[7]);
  const Pair b0 = cadd(a0, a2), b2 = csub(a0, a2);
  const Pair b1 = cadd(a1, a3), b3 = csub(a1, a3);
  const Pair b4 = cadd(a4, a6), b6 = csub_mi(a4, a6);
  const Pair t5 = cadd(a5, a7), t7 = csub(a5, a7);
  const Pair b5 = {__fmul2_rn(s, add2(t5.re, t5.im)), __fmul2_rn(s, sub2(t5.im, t5.re))};   // * exp(-i pi/4)
  const Pair b7 = {__fmul2_rn(s, sub2(t7.im, t7.re)), __fmul2_rn(ns, add2(t7.re, t7.im))};  // * exp(-3 i pi/4)
  u[0] = cadd(b0, b4);
  u[4] = csub(b0, b4);
  u[1] = cadd(b1, b5);
  u[5] = csub(b1, b5);
  u[2] = cadd(b2, b6);
  u[6] = csub(b2, b6);
  u[3] = cadd(b3, b7);
  u[7] = csub(b3, b7);
}

template <int N>
struct Radices {
  static constexpr int log2n = (N == 32) ? 5 : (N == 64) ? 6 : (N == 128) ? 7 : (N == 256) ? 8 : (N == 512) ? 9
                               : (N == 1024) ? 10 : (N == 2048) ? 11 : 12;
  static constexpr int n8 = log2n / 3;      // radix-8 stages
  static constexpr int tail = log2n % 3;    // 0, 1 (radix 2) or 2 (radix 4)
  static constexpr int stages = n8 + (tail ? 1 : 0);
};

}  // namespace fft
}  // namespace gbp
