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

// Threads of a CTA that transforms one item (INTER: N points along x, else N/2).
constexpr int x_threads(int N, bool inter) { return (inter ? N : N / 2) < 512 ? 256 : 512; }

template <int N, bool INTER, int NT_ = x_threads(N, INTER)>
struct XLayout {
  static constexpr int NX = INTER ? N : N / 2;   // points of the x transform
  static constexpr int NT = NT_;
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

// (A + B) - i f (A - B), B = conj b, f = (fr, fi): the mode (the fields come scaled, fft::PACK_SCALE).
__device__ __forceinline__ float2 unpack_mode(float2 a, float2 b, float fr, float fi) {
  const float sx = a.x + b.x, sy = a.y - b.y, dx = a.x - b.x, dy = a.y + b.y;
  return make_float2(sx + (fr * dy + fi * dx), sy + (fi * dy - fr * dx));
}

// One warp step: lane modes x0 + j (j < MS) of one column, bins monotone in
// lane order; sums runs and adds each once to the warp's bins.
template <int MS, int NV>
__device__ __forceinline__ void flush_runs(float (&P)[MS][NV], const int (&bin)[MS], int lane, float* wb, int nbe) {
  bool start[MS];
  start[0] = true;
#pragma unroll
  for (int j = 1; j < MS; ++j) {
    start[j] = bin[j] != bin[j - 1];
    if (!start[j]) {
#pragma unroll
      for (int q = 0; q < NV; ++q) P[j][q] += P[j - 1][q];
    }
  }
  bool multi = false;
#pragma unroll
  for (int j = 1; j < MS; ++j) multi = multi || start[j];
  const int prev_last = __shfl_up_sync(0xffffffffu, bin[MS - 1], 1);
  const bool cont = lane > 0 && bin[0] == prev_last;       // the lane's first run continues the previous lane's last
  const unsigned heads = __ballot_sync(0xffffffffu, multi || !cont);
  float T[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) T[q] = P[MS - 1][q];
  seg_scan<NV>(T, heads, lane);
  float Tprev[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) Tprev[q] = __shfl_up_sync(0xffffffffu, T[q], 1);
  const bool next_cont = __shfl_down_sync(0xffffffffu, cont, 1) && lane < 31;
  // runs that end inside the lane: the first of them absorbs the carry from earlier lanes
  bool carry = cont && multi;
#pragma unroll
  for (int j = 0; j < MS - 1; ++j) {
    if (start[j + 1]) {
      if (carry) {
#pragma unroll
        for (int q = 0; q < NV; ++q) P[j][q] += Tprev[q];
        carry = false;
      }
      if (bin[j] >= 0) bin_add<NV>(wb, nbe, bin[j], P[j]);
    }
  }
  if (!next_cont && bin[MS - 1] >= 0) bin_add<NV>(wb, nbe, bin[MS - 1], T);
  __syncwarp();
}

// Loads item (y, kb) of the packed spectrum `spec` (transformed over z and y)
// and transforms its 16 columns along x into s (transposed, swizzled); ends
// with a barrier.  IN_SHARED: see fft::col_fft.  W: interleaved planes
// (fft::PackedRows); W = 1: plain rows, consecutive x' `planes` planes of
// [N][P] apart (the slabs NX * planes of them).
template <int N, bool INTER, bool IN_SHARED, int NT = x_threads(N, INTER), int W = fft::PACK_W>
__device__ __forceinline__ void x_forward(float2* s, const float2* __restrict__ spec, int y, int kb,
                                          const float2* __restrict__ twx, int tid, int planes = 1) {
  using L = XLayout<N, INTER, NT>;
  using R = fft::PackedRows<N, W>;
  constexpr int TST = L::TST;
  const float2* src = spec + kb * R::BLOCK;
  // row of the column pair's slab: y, or -y of slab 1
  const long long r0 = (long long)y * R::ROW, r1 = R::plane(L::NX * planes) + (long long)((N - y) & (N - 1)) * R::ROW;
  auto gin = [src, r0, r1, planes](int x, int cp) {    // columns 2cp, 2cp+1 (slab cp / 4)
    return __ldcg(reinterpret_cast<const float4*>(src + (cp < 4 ? r0 : r1) + R::plane(x * planes)) + (cp & 3));
  };
  auto tout = [s](int x, int cp, float4 v) {
    s[(2 * cp) * TST + xswz<L::M2>(x)] = fft::lo2(v);
    s[(2 * cp + 1) * TST + xswz<L::M2>(x)] = fft::hi2(v);
  };
  fft::col_fft<L::NX, 2, L::NT, true, decltype(gin), decltype(tout), IN_SHARED>(s, gin, tout, twx, tid);
}

}  // namespace
}  // namespace gbp
