// The x pass of the packed transform (fft.cu) as the kernels that consume the
// spectrum use it: one work item = one ky row and a block of 8 adjacent kz
// columns of slab 0 (kz >= 0), and row -ky of the same block of slab 1 (-kz),
// transformed along x into shared memory, where Z(k) and Z(-k) meet.  Used by
// the binning (xbin.cu), the two-point function (xi.cu), the bispectrum
// (bispec.cu) and the gradients (grad.cu).
#pragma once

#include "fft_core.cuh"
#include "fft_pass.cuh"
#include "gbp_bins.h"
#include "gbp_fft.h"
#include "gbp_internal.cuh"
#include "power_core.cuh"

namespace gbp {
namespace {

constexpr int XB_C = 8;                      // kz columns per work item
// The next item's HBM loads start before the barrier that ends the binning (512^3 and up)
template <int N>
constexpr bool XB_EARLY = N >= 512;

template <int N, bool INTER>
struct XLayout {
  static constexpr int NX = INTER ? N : N / 2;   // points of the x transform
  static constexpr int NT = NX < 512 ? 256 : 512;
  static constexpr int HALVES = NT / 256;    // warps per column
  static constexpr int TST = NX + 1;         // complex per column (transposed layout); odd: no store conflicts
  // a lane takes M2 consecutive pairs (x, N - x) of its warp's part of the |kx| range, MS2 per warp step
  static constexpr int M2 = N / (64 * HALVES);
  static constexpr int MS2 = M2 < 4 ? M2 : (N >= 1024 && INTER ? (M2 < 8 ? M2 : 8) : 4);
  static_assert(MS2 > 0 && M2 % MS2 == 0, "whole warp steps of mode pairs");
  static __host__ __device__ constexpr size_t data_bytes() {
    const size_t rows = (size_t)2 * fft::ColBlock<NX, 2>::SLAB, cols = (size_t)2 * XB_C * TST;
    return ((rows > cols ? rows : cols) * 8 + 127) & ~size_t(127);
  }
  // per-|kx| tables (swizzled like the columns): window c2 and the factor f of kx >= 0
  static __host__ __device__ constexpr size_t xtab_bytes() { return (size_t)(N / 2) * 12; }
};

// Swizzled position of x in a transposed column: lane l reads x = base + M2 l
// + j (M2 = the mode pairs a lane takes), and so does it read the mirror
// -x; with x's low bits XORed by bits 4.. of x, the 16 lanes of a half-warp
// hit 16 distinct 8-byte slots in both reads, and the last FFT stage's
// stores stay conflict-free.
template <int M2>
__device__ __forceinline__ int xswz(int x) {
  if constexpr (M2 <= 1) return x;
  else return x ^ ((x >> 4) & (M2 - 1));
}

// (A + B) - i f (A - B), B = conj b, f = (fr, fi): four times |.|^2's root is the mode.
__device__ __forceinline__ float2 unpack_mode(float2 a, float2 b, float fr, float fi) {
  const float sx = a.x + b.x, sy = a.y - b.y, dx = a.x - b.x, dy = a.y + b.y;
  return make_float2(sx + (fr * dy + fi * dx), sy + (fi * dy - fr * dx));
}

// Loads item (y, kb) of the packed spectrum `spec` (transformed over z and y)
// and transforms its 16 columns along x into s (transposed, swizzled); ends
// with a barrier.  IN_SHARED: see fft::col_fft.
template <int N, bool INTER, bool IN_SHARED>
__device__ __forceinline__ void x_forward(float2* s, const float2* __restrict__ spec, int y, int kb,
                                          const float2* __restrict__ twx, int tid) {
  using L = XLayout<N, INTER>;
  constexpr int P = N / 2 + 8, TST = L::TST;
  const float2* src = spec + kb * XB_C;
  // row of the column pair's slab: y, or -y of slab 1
  const long long r0 = (long long)y * P, r1 = (long long)L::NX * N * P + (long long)((N - y) & (N - 1)) * P;
  auto gin = [src, r0, r1](int x, int cp) {    // columns 2cp, 2cp+1 (slab cp / 4)
    return __ldcs(reinterpret_cast<const float4*>(src + (cp < 4 ? r0 : r1) + (long long)x * N * P) + (cp & 3));
  };
  auto tout = [s](int x, int cp, float4 v) {
    s[(2 * cp) * TST + xswz<L::M2>(x)] = fft::lo2(v);
    s[(2 * cp + 1) * TST + xswz<L::M2>(x)] = fft::hi2(v);
  };
  fft::col_fft<L::NX, 2, L::NT, true, decltype(gin), decltype(tout), IN_SHARED>(s, gin, tout, twx, tid);
}

}  // namespace
}  // namespace gbp
