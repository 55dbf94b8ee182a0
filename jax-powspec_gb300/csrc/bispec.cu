// The FFT bispectrum estimator of src/correlations.py:334-462 (`bispec`):
// for shells |k| in [k_i - kF, k_i + kF) around k_1, k_2 and k_3(theta),
//
//   delta_i(x) = irfftn(mask_i W delta_k),   I_i(x) = irfftn(mask_i),
//   P_i = sum_x delta_i^2 / sum_x I_i^2 (L / N^2)^3,
//   B   = sum_x delta_1 delta_2 delta_3 / sum_x I_1 I_2 I_3 (L^2 / N^3)^3,
//   Q   = B / (P_1 P_2 + P_1 P_3 + P_2 P_3).
//
// The reference transforms two fields back per shell (2 (n_theta + 2)
// inverse FFTs).  Here Parseval's theorem moves every sum but the first two
// shells' fields to Fourier space:
//
//   sum_x delta_i^2        = N^-3 sum_k |mask_i W delta_k|^2
//   sum_x I_i^2            = N^-3 n_i                   (modes in shell i)
//   sum_x delta_1 delta_2 delta_3 = N^-3 sum_k mask_3 W delta_k conj(FFT(delta_1 delta_2))
//   sum_x I_1 I_2 I_3      = N^-3 sum_k mask_3 conj(FFT(I_1 I_2))
//
// so a whole theta scan costs four inverse transforms (delta_1, delta_2,
// I_1, I_2), two forward transforms (of the products delta_1 delta_2 and
// I_1 I_2) and one pass over the spectrum that bins every mode once:
//
//   1. R2C of the contrast (the plan's transform) into the caller's spectrum,
//   2. bispec_fill_kernel: mask_1 W delta_k, mask_2 W delta_k, mask_1, mask_2
//      as four half spectra,
//   3. one batched cuFFT C2R of the four (unnormalised; the common factor
//      N^3 cancels in every ratio),
//   4. bispec_products_kernel: delta_1 delta_2 and I_1 I_2, in place,
//   5. the plan's R2C of the two products,
//   6. bispec_bin_kernel: every half-spectrum mode with its Hermitian weight
//      (2, or 1 on the kz = 0 and Nyquist planes) into elementary bins --
//      the intervals between consecutive shell limits, so that every shell
//      is a run of them -- with four sums: w |W delta|^2, w W Re(delta
//      conj D), w Re J, w; per-warp float32 bins, float-float partials,
//   7. bispec_reduce_kernel: the partials in double, in a fixed order,
//   8. bispec_finish_kernel: shell sums from their elementary bins, P, B, Q.
//
// For the library's transform sizes the same sums come from the packed
// transform (fft.cu), pruned to the shells at every pass, without cuFFT:
//
//   a. z, y pass of the contrast (gbp_fft_power's), kept up to the last shell,
//   b. bispec_x_kernel: x pass of an item, then the inverse x transforms of
//      a(k) = W delta_k (mask_1 + i mask_2) at (ky, kz) and (-ky, -kz), and of
//      the (real, even) b(k) = mask_1 + i mask_2 at (ky, kz),
//   c. inverse y pass of a and b (rows outside shells 1 and 2 are zeros),
//   d. bispec_z_kernel: inverse z transforms of a pencil of a and b, which are
//      delta_1 + i delta_2 and I_1 + i I_2, their products delta_1 delta_2 and
//      I_1 I_2, and the z pass of both, packed as one grid is (x planes 2x',
//      2x'+1 together; packing the two products together would round one to
//      the other's magnitude), all in shared memory; the products' spectra
//      take the even and the odd planes of slabs 0 and 1,
//   e. y pass of both,
//   f. bispec_xbin_kernel: x passes of an item of the contrast and of both
//      products, and the four sums, binned as in xbin.cu.
//
// 256^3, k1 = 0.1, k2 = 0.2, 20 angles, L = 2500: 0.857 -> 0.43 ms of kernels (x 0.050, y 0.051, z 0.101,
// x + bins 0.116).
//
// Shell membership is the reference's float32 rule, k = sqrtf(k^2) >=
// (k_i - kF) / kF and < (k_i + kF) / kF, through the bin plan's integer k^2
// thresholds.  Deterministic: no float atomics.
#include <cufft.h>
#include <limits.h>
#include <math.h>

#include <algorithm>

#include "xpass.cuh"

namespace gbp {
namespace {

constexpr int BK_NV = 4;   // w |W delta|^2, w W Re(delta conj D), w Re J, w

// Amplitude window of one axis, sinc^(-p) = (1/sinc^2)^(p/2).
__device__ __forceinline__ float amp_axis(float inv_sinc2, int p) {
  float a = 1.0f;
  for (int i = 0; i < (p >> 1); ++i) a *= inv_sinc2;
  if (p & 1) a *= sqrtf(inv_sinc2);
  return a;
}

// k^2 threshold of elementary edge e: modes with k^2 >= it are at or above the edge.
__device__ __forceinline__ int edge_q(const int* __restrict__ thr, int nbe, int e) {
  if (e <= 0) return e < 0 ? 0 : __ldg(thr);
  return e <= nbe ? __ldg(thr + e) : INT_MAX;      // edges past nbe are beyond every mode
}

__global__ void bispec_fill_kernel(const float2* __restrict__ spec, int P, float2* __restrict__ A, int Pc, int N,
                                   const int* __restrict__ thr, int nbe, const int* __restrict__ shell_bins,
                                   const float* __restrict__ inv_sinc2, int p) {
  const long long T = (long long)N * N * Pc;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  const int kz = (int)(i % Pc);
  const long long row = i / Pc;
  const int iy = (int)(row % N), ix = (int)(row / N);
  const int kx = signed_k(ix, N), ky = signed_k(iy, N);
  const int k2 = kx * kx + ky * ky + kz * kz;
  const bool m1 = k2 >= edge_q(thr, nbe, __ldg(shell_bins + 0)) && k2 < edge_q(thr, nbe, __ldg(shell_bins + 1));
  const bool m2 = k2 >= edge_q(thr, nbe, __ldg(shell_bins + 2)) && k2 < edge_q(thr, nbe, __ldg(shell_bins + 3));
  float2 v1 = make_float2(0.f, 0.f), v2 = v1;
  if (m1 || m2) {
    const float c = amp_axis(__ldg(inv_sinc2 + abs(kx)), p) * amp_axis(__ldg(inv_sinc2 + abs(ky)), p) *
                    amp_axis(__ldg(inv_sinc2 + kz), p);
    const float2 d = spec[row * P + kz];
    const float2 cd = make_float2(d.x * c, d.y * c);
    if (m1) v1 = cd;
    if (m2) v2 = cd;
  }
  A[i] = v1;
  A[T + i] = v2;
  A[2 * T + i] = make_float2(m1 ? 1.f : 0.f, 0.f);
  A[3 * T + i] = make_float2(m2 ? 1.f : 0.f, 0.f);
}

// R[0] <- R[0] R[1], R[1] <- R[2] R[3] (fields of M cells each).
__global__ void bispec_products_kernel(float* R, long long M) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  if ((M & 3) == 0) {
    float4* r4 = reinterpret_cast<float4*>(R);
    const long long M4 = M >> 2;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M4; i += stride) {
      const float4 a = r4[i], b = r4[M4 + i], c = r4[2 * M4 + i], d = r4[3 * M4 + i];
      r4[i] = make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
      r4[M4 + i] = make_float4(c.x * d.x, c.y * d.y, c.z * d.z, c.w * d.w);
    }
  } else {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < M; i += stride) {
      const float a = R[i], b = R[M + i], c = R[2 * M + i], d = R[3 * M + i];
      R[i] = a * b;
      R[M + i] = c * d;
    }
  }
}

// One warp step over 32 consecutive entries of the [N][N][P] spectra.
__device__ __forceinline__ void bk_step(const PowGeom& g, const Smem& t, const float2* __restrict__ sd,
                                        const float2* __restrict__ sD, const float2* __restrict__ sJ, float* wb,
                                        int lane, long long f, long long end) {
  const int N = g.N, P = g.Lzs, h = N / 2;
  const int kz = (int)(f % P);
  const long long row = f / P;
  float v[BK_NV] = {0.f, 0.f, 0.f, 0.f};
  int bin = -1;
  if (f < end && kz <= h) {
    const int iy = (int)(row % N), ix = (int)(row / N);
    const int kx = signed_k(ix, N), ky = signed_k(iy, N);
    bin = bin_of(g, t, kx * kx + ky * ky + kz * kz);
    if (bin >= 0) {
      const float c = t.c2[kx < 0 ? -kx : kx] * t.c2[ky < 0 ? -ky : ky] * t.c2[kz];
      const float w = (kz == 0 || ((N & 1) == 0 && kz == h)) ? 1.0f : 2.0f;
      const float2 d = sd[f], D = sD[f], J = sJ[f];
      const float dr = d.x * c, di = d.y * c;
      v[0] = w * (dr * dr + di * di);
      v[1] = w * (dr * D.x + di * D.y);
      v[2] = w * J.x;
      v[3] = w;
    }
  }
  const long long rprev = __shfl_up_sync(0xffffffffu, row, 1);
  const int bprev = __shfl_up_sync(0xffffffffu, bin, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || bin != bprev || row != rprev);
  seg_scan<BK_NV>(v, heads, lane);
  const bool segend = (lane == 31) || ((heads >> (lane + 1)) & 1u);
  // runs of different z rows in one step may share a bin: flush row by row
  const int rel = (int)(row - __shfl_sync(0xffffffffu, row, 0));
  const int nph = __reduce_max_sync(0xffffffffu, f < end ? rel : 0) + 1;
  for (int ph = 0; ph < nph; ++ph) {
    if (segend && bin >= 0 && rel == ph) bin_add<BK_NV>(wb, g.nbe, bin, v);
    __syncwarp();
  }
}

__global__ void __launch_bounds__(POW_WARPS * 32, 4)
bispec_bin_kernel(PowGeom g, const float2* __restrict__ sD, const float2* __restrict__ sJ, int p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const Smem s = load_tables<BK_NV, false>(g, smem);          // g.mas_order = 0: c2 is rewritten below
  for (int k = threadIdx.x; k <= g.N / 2; k += blockDim.x) s.c2[k] = amp_axis(g.inv_sinc2[k], p);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* wb = s.wbase + warp * BK_NV * g.nbe;
  for (int grp = blockIdx.x; grp < g.groups; grp += gridDim.x) {
    const long long beg = ((long long)grp * g.warps + warp) * g.chunk;
    const long long end = min(beg + g.chunk, g.total);
    for (long long f = beg + lane; f - lane < end; f += 32) bk_step(g, s, g.s0, sD, sJ, wb, lane, f, end);
    cta_fold<BK_NV>(g, s, grp);
  }
}

// ---- packed path (library transform sizes) ---------------------------------
struct ShellLimits {
  int q[4];      // shells 1 and 2: k^2 in [q[0], q[1]) and [q[2], q[3])
  int lim;       // the largest k^2 of either, at most k2_max
};

__device__ __forceinline__ ShellLimits shell_limits(const int* __restrict__ thr, int nbe,
                                                    const int* __restrict__ shell_bins, int k2_max) {
  ShellLimits s;
#pragma unroll
  for (int i = 0; i < 4; ++i) s.q[i] = edge_q(thr, nbe, __ldg(shell_bins + i));
  s.lim = min(k2_max, max(s.q[1], s.q[3]) - 1);
  return s;
}

__device__ __forceinline__ float2 shell_mask(const ShellLimits& s, int k2) {
  return make_float2(k2 >= s.q[0] && k2 < s.q[1] ? 1.f : 0.f, k2 >= s.q[2] && k2 < s.q[3] ? 1.f : 0.f);
}

template <int N>
struct BxLayout {
  using L = XLayout<N, false>;
  static constexpr int NT = L::NT;
  static constexpr size_t DATA = ((size_t)2 * fft::ColBlock<N, 2>::SLAB * 8 + 127) & ~size_t(127);
  static_assert(DATA >= L::data_bytes(), "the forward transform fits the inverse one's buffer");
  static constexpr size_t SMEM = DATA + (size_t)(N / 2 + 1) * sizeof(float);
};

// a into slabs 0 (ky, kz) and 1 (-ky, -kz) of out, b into slab 2, for the
// items that reach shell 1 or 2.
template <int N>
__global__ void __launch_bounds__(BxLayout<N>::NT, N >= 512 ? 1 : 3)
bispec_x_kernel(PowGeom g, const int* __restrict__ shell_bins, int k2_max, int p, float2* __restrict__ out) {
  pdl_wait();
  using L = XLayout<N, false>;
  constexpr int P = N / 2 + 8, TST = L::TST, NX = L::NX, NT = L::NT, H = N / 2;
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = reinterpret_cast<float2*>(smem);
  float* c2 = reinterpret_cast<float*>(smem + BxLayout<N>::DATA);
  const int tid = threadIdx.x;
  const ShellLimits sl = shell_limits(g.thr, g.nbe, shell_bins, k2_max);
  for (int k = tid; k <= H; k += NT) c2[k] = amp_axis(g.inv_sinc2[k], p);
  __syncthreads();
  const long long sstride = (long long)N * N * P;
  for (int it = blockIdx.x; it < g.items; it += gridDim.x) {
    const int y = it / (P / 8), kb = it - y * (P / 8);
    const int ky = signed_k(y, N), ay = ky < 0 ? -ky : ky;
    if (ky * ky + 64 * kb * kb > sl.lim) continue;           // uniform over the block
    x_forward<N, false, false>(s, g.s0, y, kb, g.twx, tid);
    // W delta_k (mask_1 + i mask_2) of column c at kx = x (slab 0), or at -(kx = -x) (slab 1), re and im swapped
    auto value = [&](int x, int c, int slab) {
      const int kz = kb * XB_C + c;
      if (kz > H) return make_float2(0.f, 0.f);
      const int kx = signed_k(x, N), ax = kx < 0 ? -kx : kx;
      const float2 m = shell_mask(sl, kx * kx + ky * ky + kz * kz);
      if (m.x + m.y == 0.f) return make_float2(0.f, 0.f);
      const int xk = slab ? (N - x) & (N - 1) : x;           // the mode of (ky, kz) it comes from
      const float2 w = __ldg(g.tw + xk);
      const float2 d = unpack_mode(s[c * TST + xswz<L::M2>(xk & (NX - 1))],
                                   s[(XB_C + c) * TST + xswz<L::M2>((NX - xk) & (NX - 1))], w.x, w.y);
      const float f = c2[ax] * c2[ay] * c2[kz];
      const float dr = d.x * f, di = slab ? -d.y * f : d.y * f;
      return make_float2(dr * m.y + di * m.x, dr * m.x - di * m.y);
    };
    auto gin = [&](int x, int cp) {
      const float2 u = value(x, 2 * (cp & 3), cp >> 2), v = value(x, 2 * (cp & 3) + 1, cp >> 2);
      return make_float4(u.x, u.y, v.x, v.y);
    };
    float2* dst = out + kb * XB_C;
    const long long r0 = (long long)y * P, r1 = sstride + (long long)((N - y) & (N - 1)) * P;
    auto gout = [dst, r0, r1](int x, int cp, float4 v) {
      __stcs(reinterpret_cast<float4*>(dst + (cp < 4 ? r0 : r1) + (long long)x * N * P) + (cp & 3),
             make_float4(v.y, v.x, v.w, v.z));
    };
    fft::col_fft<N, 2, NT, false, decltype(gin), decltype(gout), true>(s, gin, gout, g.tw, tid);
    // b is even along every axis: its forward and inverse transforms agree
    auto bin_ = [&](int x, int cp) {
      const int kx = signed_k(x, N), kp = kx * kx + ky * ky, kz = kb * XB_C + 2 * cp;
      const float2 z = make_float2(0.f, 0.f);
      const float2 u = kz <= H ? shell_mask(sl, kp + kz * kz) : z;
      const float2 v = kz < H ? shell_mask(sl, kp + (kz + 1) * (kz + 1)) : z;
      return make_float4(u.x, u.y, v.x, v.y);
    };
    auto bout = [dst, r0, sstride](int x, int cp, float4 v) {
      __stcs(reinterpret_cast<float4*>(dst + 2 * sstride + r0 + (long long)x * N * P) + cp, v);
    };
    fft::col_fft<N, 1, NT, false, decltype(bin_), decltype(bout), true>(s, bin_, bout, g.tw, tid);
    __syncthreads();
  }
}

// Inverse y pass of the three slabs: rows and kz blocks outside shells 1 and 2 hold nothing.
template <int N>
__global__ void __launch_bounds__(N / 2, N <= 512 ? 4 : 2)
bispec_y_kernel(PowGeom g, const int* __restrict__ shell_bins, int k2_max, int nkb, float2* __restrict__ data) {
  pdl_wait();
  constexpr int P = N / 2 + 8;
  extern __shared__ __align__(16) float2 sy[];
  const int plane = blockIdx.x / nkb, kb = blockIdx.x % nkb;
  const int lim = shell_limits(g.thr, g.nbe, shell_bins, k2_max).lim - 64 * kb * kb;
  if (lim < 0) return;
  float2* base = data + (long long)plane * N * P + kb * 8;
  auto gin = [base, lim](int j, int cp) {
    const int k = signed_k(j, N);
    if (k * k > lim) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v = __ldcg(reinterpret_cast<const float4*>(base + (long long)j * P) + cp);
    return make_float4(v.y, v.x, v.w, v.z);
  };
  auto gout = [base](int j, int cp, float4 v) {
    __stcs(reinterpret_cast<float4*>(base + (long long)j * P) + cp, make_float4(v.y, v.x, v.w, v.z));
  };
  fft::col_fft<N, 1, N / 2, false>(sy, gin, gout, g.tw, threadIdx.x);
}

// Column stages whose barriers cover the threads of a column pair, or a warp (bispec_z at 256^3: 0.106 -> 0.101 ms).
template <int N, int CP, int NT, bool IN_SHARED, bool OUT_SHARED, class GIn, class SIn, class SOut, class GOut>
__device__ __forceinline__ void bz_stages(GIn gin, SIn sin_, SOut sout, GOut gout, const float2* __restrict__ tw,
                                          int tid) {
  fft::run_stages2<N, CP, NT, true, IN_SHARED, OUT_SHARED, GIn, SIn, SOut, GOut, fft::GROUP<N>>(gin, sin_, sout, gout,
                                                                                            tw, tid);
}

// PAIRS pencils per CTA (two x planes, PAIRS / 2 rows): a and b back along z,
// products, forward along z into the pencils' own rows of slabs 0 and 1 (read
// before they are written): plane 2x' for delta_1 delta_2, 2x'+1 for I_1 I_2.
template <int N, int PAIRS>
__global__ void __launch_bounds__(PAIRS * N / 16)
bispec_z_kernel(PowGeom g, const int* __restrict__ shell_bins, int k2_max, int kz_cols, float2* __restrict__ data) {
  pdl_wait();
  constexpr int NT = PAIRS * N / 16, CP = PAIRS / 2, P = N / 2 + 8, H = N / 2;
  static_assert(N % CP == 0, "a block's rows share one pair of planes");
  extern __shared__ __align__(16) float4 sz[];               // a and b, [CP][N] slots of two pencils each
  float4* sb = sz + CP * N;
  const int tid = threadIdx.x;
  const int lim = shell_limits(g.thr, g.nbe, shell_bins, k2_max).lim;
  const long long sstride = (long long)N * N * P, pstride = (long long)N * P;
  const int xp = blockIdx.x / (N / CP), y0 = (blockIdx.x - xp * (N / CP)) * CP;
  float2* i0 = data + (long long)2 * xp * pstride + (long long)y0 * P;
  float2* i1 = i0 + sstride;
  const float2* i2 = i0 + 2 * sstride;
  auto load = [lim, pstride](const float2* row, int k, int cp) {   // row y0 + cp of planes 2x', 2x'+1
    if (64 * (k >> 3) * (k >> 3) > lim) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 u = __ldcg(row + cp * P + k), v = __ldcg(row + pstride + cp * P + k);
    return make_float4(u.x, u.y, v.x, v.y);
  };
  auto agin = [&](int j, int cp) {
    const float4 v = j <= H ? load(i0, j, cp) : load(i1, N - j, cp);
    return make_float4(v.y, v.x, v.w, v.z);
  };
  auto bgin = [&](int j, int cp) { return load(i2, j <= H ? j : N - j, cp); };
  auto asin = [sz_ = sz](int j, int cp) { return sz_[cp * N + fft::zsw(j)]; };
  auto asout = [sz_ = sz](int j, int cp, float4 v) { sz_[cp * N + fft::zsw(j)] = v; };
  auto bsin = [sb](int j, int cp) { return sb[cp * N + fft::zsw(j)]; };
  auto bsout = [sb](int j, int cp, float4 v) { sb[cp * N + fft::zsw(j)] = v; };
  bz_stages<N, CP, NT, false, true>(agin, asin, asout, asout, g.tw, tid);
  bz_stages<N, CP, NT, false, true>(bgin, bsin, bsout, bsout, g.tw, tid);
  // one column of each product per row (the swapped parts of a multiply to the same)
  auto cgin = [&](int j, int cp) {
    const float4 a = asin(j, cp), b = bsin(j, cp);
    return make_float4(a.x * a.y, a.z * a.w, b.x * b.y, b.z * b.w);
  };
  auto cgout = [i0, i1, kz_cols, pstride](int k, int cp, float4 v) {
    const int m = (N - k) & (N - 1);
    if (k <= H && k < kz_cols) {
      __stcs(i0 + cp * P + k, fft::lo2(v));
      __stcs(i0 + pstride + cp * P + k, fft::hi2(v));
    }
    if (m <= H && m < kz_cols) {
      __stcs(i1 + cp * P + m, fft::lo2(v));
      __stcs(i1 + pstride + cp * P + m, fft::hi2(v));
    }
  };
  bz_stages<N, CP, NT, true, false>(cgin, asin, asout, cgout, g.tw, tid);
}

template <int N>
struct BbLayout {
  static constexpr int NT = x_threads(N, true);
  using L = XLayout<N, false, NT>;               // the contrast's columns, then each product's
  static constexpr int MS = L::M2 < 2 ? L::M2 : 2;
  static constexpr size_t DATA = 3 * L::data_bytes();
};

// The four sums of the pairs of modes kx = +-p, p = p0 .. p0 + MS - 1, of one
// column (a at (ky, kz), b = a + XB_C TST at (-ky, -kz)) of the contrast and
// the products, `field` complex apart.
template <int N, int MS>
__device__ __forceinline__ void bispec_pairs(const PowGeom& g, const Smem& t, const float2* a, int field, int p0,
                                             int kyz2, float cyz, float w, float (&v)[MS][BK_NV], int (&bin)[MS]) {
  using L = typename BbLayout<N>::L;
  const float2* b = a + XB_C * L::TST;
#pragma unroll
  for (int j = 0; j < MS; ++j) {
    const int p = p0 + j, k2 = p * p + kyz2;
    bin[j] = bin_of(g, t, k2);
    const int sp = xswz<L::M2>(p & (L::NX - 1)), sm = xswz<L::M2>((L::NX - p) & (L::NX - 1));
    const float2 e = __ldg(g.tw + p);
    const float c = cyz * t.c2[p];               // of d; D and J, unscaled fields, come out twice the mode
    float q[BK_NV] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; ++h) {                // kx = p, then kx = -p (the same mode when p = 0 or N/2)
      if (h == 1 && (p == 0 || p == N / 2)) break;
      const int sa = h ? sm : sp, sn = h ? sp : sm;
      const float ei = h ? -e.y : e.y;
      const float2 d = unpack_mode(a[sa], b[sn], e.x, ei);
      const float2 D = unpack_mode(a[field + sa], b[field + sn], e.x, ei);
      const float2 J = unpack_mode(a[2 * field + sa], b[2 * field + sn], e.x, ei);
      q[0] += d.x * d.x + d.y * d.y;
      q[1] += d.x * D.x + d.y * D.y;
      q[2] += J.x;
      q[3] += 1.0f;
    }
    v[j][0] = w * q[0] * (c * c);
    v[j][1] = w * q[1] * (0.5f * c);
    v[j][2] = w * q[2] * 0.5f;
    v[j][3] = w * q[3];
  }
}

template <int N>
__global__ void __launch_bounds__(BbLayout<N>::NT, N >= 1024 ? 1 : 2)
bispec_xbin_kernel(PowGeom g, const float2* __restrict__ pair, int k2_max, int p) {
  pdl_wait();
  using B = BbLayout<N>;
  using L = typename B::L;
  constexpr int P = N / 2 + 8, NT = B::NT, H = N / 2, HALVES = L::HALVES, M2 = L::M2, MS = B::MS;
  constexpr int FIELD = (int)(L::data_bytes() / sizeof(float2));
  extern __shared__ __align__(16) unsigned char smem[];
  float2* sd = reinterpret_cast<float2*>(smem);
  const Smem t = load_tables<BK_NV, false>(g, smem + B::DATA);          // g.mas_order = 0: c2 is rewritten below
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int k = tid; k <= H; k += NT) t.c2[k] = amp_axis(g.inv_sinc2[k], p);
  __syncthreads();
  for (int grp = blockIdx.x; grp < g.groups; grp += gridDim.x) {
    for (int it = grp; it < g.items; it += g.groups) {
      const int y = it / (P / 8), kb = it - y * (P / 8);
      const int ky = signed_k(y, N), ay = ky < 0 ? -ky : ky;
      if (ky * ky + 64 * kb * kb > k2_max) continue;                     // uniform over the block
      x_forward<N, false, false, NT>(sd, g.s0, y, kb, g.twx, tid);
      x_forward<N, false, false, NT, 1>(sd + FIELD, pair, y, kb, g.twx, tid, 2);
      x_forward<N, false, false, NT, 1>(sd + 2 * FIELD, pair + (long long)N * P, y, kb, g.twx, tid, 2);
      const int c = warp / HALVES, h = warp % HALVES, kz = kb * XB_C + c;
      const bool active = kz <= H;
      const int kzc = active ? kz : 0;
      const float cyz = t.c2[ay] * t.c2[kzc], w = (kzc == 0 || kzc == H) ? 1.0f : 2.0f;
      const int kyz2 = ky * ky + kzc * kzc;
      const float2* a = sd + c * L::TST;
      float* wb = t.wbase + (warp & 7) * BK_NV * g.nbe;
#pragma unroll 1
      for (int s0 = 0; s0 < M2; s0 += MS) {
        float v[MS][BK_NV];
        int bin[MS];
        if (active)
          bispec_pairs<N, MS>(g, t, a, FIELD, h * (H / HALVES) + lane * M2 + s0, kyz2, cyz, w, v, bin);
        auto flush = [&]() {
          flush_runs<MS, BK_NV>(v, bin, lane, wb, g.nbe);
          if (h == HALVES - 1 && s0 + MS >= M2 && (H * H + kyz2 <= k2_max)) {
            if (lane == 0) {                                              // the mode kx = N/2
              float vn[1][BK_NV];
              int bn[1];
              bispec_pairs<N, 1>(g, t, a, FIELD, H, kyz2, cyz, w, vn, bn);
              if (bn[0] >= 0) bin_add<BK_NV>(wb, g.nbe, bn[0], vn[0]);
            }
            __syncwarp();
          }
        };
        if constexpr (HALVES == 1) {
          if (active) flush();
        } else {                                                          // two warps per bin array, in turn
          if (warp < 8 && active) flush();
          __syncthreads();
          if (warp >= 8 && active) flush();
          __syncthreads();
        }
      }
      __syncthreads();
    }
    cta_fold<BK_NV>(g, t, grp);
  }
}

struct BpLayout {
  int k2_max, kz_cols, items, groups;
  size_t smem_x, smem_b, data, part, E, total_ws;
};

template <int N>
int bp_layout_n(const gbp_bins_s* B, BpLayout& L) {
  L.smem_x = BxLayout<N>::SMEM;
  L.smem_b = BbLayout<N>::DATA + smem_plan(N, B->nbe, B->lut_n, 8, BK_NV).total;
  return L.smem_x > 227 * 1024 || L.smem_b > 227 * 1024 ? GBP_ERR_UNSUPPORTED : GBP_OK;
}

// GBP_ERR_UNSUPPORTED: the plan or the bins need the cuFFT path.
int bp_layout(const gbp_fft_plan_s* plan, const gbp_bins_s* B, BpLayout& L) {
  if (!plan->own) return GBP_ERR_UNSUPPORTED;
  const int N = plan->n, P = plan->pitch;
  int st = GBP_ERR_UNSUPPORTED;
  switch (N) {
    case 64: st = bp_layout_n<64>(B, L); break;
    case 128: st = bp_layout_n<128>(B, L); break;
    case 256: st = bp_layout_n<256>(B, L); break;
    case 512: st = bp_layout_n<512>(B, L); break;
    case 1024: st = bp_layout_n<1024>(B, L); break;
  }
  if (st) return st;
  L.k2_max = B->last_closed;      // shells may take in the last elementary bin
  L.kz_cols = 0;
  for (int kb = 0; 8 * kb <= N / 2 && 64LL * kb * kb <= L.k2_max; ++kb) L.kz_cols = 8 * (kb + 1);
  L.items = N * (P / 8);
  L.groups = std::min(L.items, 1216);
  L.data = align256((size_t)3 * N * N * P * sizeof(float2));
  L.part = align256((size_t)L.groups * BK_NV * B->nbe * sizeof(float2));
  L.E = align256((size_t)B->nbe * BK_NV * sizeof(double));
  L.total_ws = L.data + L.part + L.E;
  return GBP_OK;
}

template <int N>
int run_bispec_packed(gbp_fft_plan plan, PowGeom g, const BpLayout& L, const int32_t* shell_bins, int mas_order,
                      float2* data, cudaStream_t st) {
  constexpr int PAIRS = N >= 256 ? 8 : 32768 / (N * 8);
  const float2* pair = data;
  if (L.kz_cols > 0) {
    {
      auto k = bispec_x_kernel<N>;
      GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem_x));
      GBP_TRACE("bispec_x", st);
      GBP_CUDA_TRY(launch_pdl(k, dim3(L.groups), dim3(BxLayout<N>::NT), L.smem_x, st, g, shell_bins, L.k2_max,
                              mas_order, data));
    }
    {
      const size_t smem = (size_t)fft::ColBlock<N, 1>::SLAB * sizeof(float2);
      auto k = bispec_y_kernel<N>;
      GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      GBP_TRACE("bispec_y", st);
      GBP_CUDA_TRY(launch_pdl(k, dim3(3 * N * (L.kz_cols / 8)), dim3(N / 2), smem, st, g, shell_bins, L.k2_max,
                              L.kz_cols / 8, data));
    }
    {
      const size_t smem = (size_t)2 * PAIRS * N * sizeof(float2);
      auto k = bispec_z_kernel<N, PAIRS>;
      GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      GBP_TRACE("bispec_z", st);
      GBP_CUDA_TRY(launch_pdl(k, dim3(N * N / PAIRS), dim3(PAIRS * N / 16), smem, st, g, shell_bins, L.k2_max,
                              L.kz_cols, data));
    }
    const int r = own_fft_y_rows(N, 2 * N, data, L.kz_cols, L.k2_max, plan->tw, st);
    if (r) return r;
  }
  auto k = bispec_xbin_kernel<N>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem_b));
  GBP_TRACE("bispec_bins", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3(L.groups), dim3(BbLayout<N>::NT), L.smem_b, st, g, pair, L.k2_max, mas_order));
  return GBP_OK;
}

// One block per elementary bin: the C group partials folded in a fixed order (fold_bin).
__global__ void __launch_bounds__(FOLD_THREADS)
bispec_reduce_kernel(const float2* __restrict__ part_ff, int C, int nbe, double* E) {
  pdl_wait();
  const int b = blockIdx.x;
  if (b >= nbe) return;                        // uniform over the block
  double m[BK_NV] = {0.0, 0.0, 0.0, 0.0};
  fold_bin<BK_NV>(part_ff, C, BK_NV, nbe, b, m);
  if (threadIdx.x == 0)
    for (int q = 0; q < BK_NV; ++q) E[b * BK_NV + q] = m[q];
}

struct ShellSums {
  double p, b, t, n;
};

__device__ ShellSums shell_sums(const double* __restrict__ E, int nbe, const int* __restrict__ shell_bins, int s) {
  const int lo = max(0, shell_bins[2 * s]), hi = min(nbe, shell_bins[2 * s + 1]);
  ShellSums r{0.0, 0.0, 0.0, 0.0};
  for (int e = lo; e < hi; ++e) {
    r.p += E[e * BK_NV + 0];
    r.b += E[e * BK_NV + 1];
    r.t += E[e * BK_NV + 2];
    r.n += E[e * BK_NV + 3];
  }
  return r;
}

__global__ void bispec_finish_kernel(const double* __restrict__ E, int nbe, const int* __restrict__ shell_bins,
                                     int S, int N, double box, double* pk_out, double* bk_out, double* qk_out,
                                     long long* nmodes_out) {
  pdl_wait();
  const double n3 = (double)N * N * N;
  const double pnorm = (box / ((double)N * N)) * (box / ((double)N * N)) * (box / ((double)N * N));
  const double l2n3 = box * box / n3;
  const double bnorm = l2n3 * l2n3 * l2n3;
  const ShellSums a = shell_sums(E, nbe, shell_bins, 0), b = shell_sums(E, nbe, shell_bins, 1);
  const double p1 = a.p / a.n * pnorm, p2 = b.p / b.n * pnorm;
  for (int s = threadIdx.x; s < S; s += blockDim.x) {
    const ShellSums r = s == 0 ? a : (s == 1 ? b : shell_sums(E, nbe, shell_bins, s));
    const double p3 = r.p / r.n * pnorm;
    pk_out[s] = p3;
    if (nmodes_out) nmodes_out[s] = (long long)llrint(r.n);
    if (s >= 2) {
      const double bk = r.b / r.t * bnorm;
      bk_out[s - 2] = bk;
      qk_out[s - 2] = bk / (p1 * p2 + p1 * p3 + p2 * p3);
    }
  }
}

struct BkLayout {
  int warps, C, Pc;
  long long total, chunk;
  size_t smem, A, R, part, E, cws, total_ws;
};

int bk_layout(const gbp_fft_plan_s* plan, const gbp_bins_s* B, BkLayout& L) {
  const int N = plan->n;
  int w = POW_WARPS;
  while (w > 1 && smem_plan(N, B->nbe, B->lut_n, w, BK_NV).total > 200 * 1024) --w;
  L.smem = smem_plan(N, B->nbe, B->lut_n, w, BK_NV).total;
  if (L.smem > 200 * 1024) return GBP_ERR_UNSUPPORTED;
  L.warps = w;
  L.Pc = N / 2 + 1;
  L.total = (long long)N * N * plan->pitch;
  long long target = L.total / (8LL * 152 * 8);
  target = std::max(1024LL, std::min(16384LL, target));
  L.chunk = (target + 31) & ~31LL;
  const long long nw = (L.total + L.chunk - 1) / L.chunk;
  L.C = (int)((nw + w - 1) / w);
  const size_t M = (size_t)N * N * N;
  // the four half spectra; the two product spectra later reuse the same bytes
  L.A = align256(std::max((size_t)4 * N * N * L.Pc, (size_t)2 * N * N * plan->pitch) * sizeof(float2));
  L.R = align256(4 * M * sizeof(float));
  L.part = align256((size_t)L.C * BK_NV * B->nbe * sizeof(float2));
  L.E = align256((size_t)B->nbe * BK_NV * sizeof(double));
  cufftHandle h;
  size_t cw = 0;
  const int st = c2r_plan(N, L.Pc, 4, &h, &cw);
  if (st) return st;
  L.cws = align256(std::max(std::max(cw, plan->ws), (size_t)1));
  L.total_ws = L.A + L.R + L.part + L.E + L.cws;
  return GBP_OK;
}

PowGeom bk_geom(const gbp_fft_plan_s* plan, const gbp_bins_s* B, const void* spectrum, float2* part) {
  PowGeom g{};
  g.s0 = static_cast<const float2*>(spectrum);
  g.N = plan->n;
  g.Lz = plan->n / 2 + 1;
  g.Lzs = plan->pitch;
  g.nb = B->nb;
  g.nbe = B->nbe;
  g.tu = B->last_closed;
  g.lut_shift = B->lut_shift;
  g.lut_n = B->lut_n;
  g.mas_order = 0;
  g.thr = B->d_thr;
  g.lut = B->d_lut;
  g.inv_sinc2 = B->d_inv_sinc2;
  g.eph = B->d_eph;
  g.part_ff = part;
  return g;
}

// Partials -> P, B, Q per shell.
int bispec_outputs(const gbp_bins_s* B, const float2* part, int groups, double* E, const int32_t* shell_bins,
                   int n_shells, int N, double box_size, double* pk_out, double* bk_out, double* qk_out,
                   long long* nmodes_out, cudaStream_t st) {
  {
    GBP_TRACE("bispec_reduce", st);
    GBP_CUDA_TRY(launch_pdl(bispec_reduce_kernel, dim3(B->nbe), dim3(FOLD_THREADS), 0, st, part, groups, B->nbe, E));
  }
  GBP_TRACE("bispec_finish", st);
  GBP_CUDA_TRY(launch_pdl(bispec_finish_kernel, dim3(1), dim3(256), 0, st, static_cast<const double*>(E), B->nbe,
                          shell_bins, n_shells, N, box_size, pk_out, bk_out, qk_out, nmodes_out));
  return GBP_OK;
}

int bispec_packed(gbp_fft_plan plan, const float* delta, void* spectrum, const gbp_bins_s* B, int mas_order,
                  const int32_t* shell_bins, int n_shells, double box_size, double* pk_out, double* bk_out,
                  double* qk_out, long long* nmodes_out, void* workspace, size_t ws_bytes, const BpLayout& L,
                  cudaStream_t st) {
  if (((reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(spectrum)) & 15u) != 0) return GBP_ERR_INVALID;
  if (!workspace || ws_bytes < L.total_ws) return GBP_ERR_WORKSPACE;
  const int N = plan->n;
  Carver cv(workspace);
  float2* data = cv.take<float2>(L.data / sizeof(float2));
  float2* part = cv.take<float2>(L.part / sizeof(float2));
  double* E = cv.take<double>(L.E / sizeof(double));
  float2* spec = static_cast<float2*>(spectrum);
  int r;
  if (L.kz_cols > 0) {
    r = own_fft_z_packed(N, 1, delta, spec, L.kz_cols, plan->tw, st);
    if (r) return r;
    r = own_fft_y_packed(N, 1, spec, L.kz_cols, L.k2_max, plan->tw, st);
    if (r) return r;
  }
  PowGeom g = bk_geom(plan, B, spec, part);
  g.tw = plan->tw;
  g.twx = plan->twx;
  g.warps = 8;
  g.items = L.items;
  g.groups = L.groups;
  switch (N) {
    case 64: r = run_bispec_packed<64>(plan, g, L, shell_bins, mas_order, data, st); break;
    case 128: r = run_bispec_packed<128>(plan, g, L, shell_bins, mas_order, data, st); break;
    case 256: r = run_bispec_packed<256>(plan, g, L, shell_bins, mas_order, data, st); break;
    case 512: r = run_bispec_packed<512>(plan, g, L, shell_bins, mas_order, data, st); break;
    default: r = run_bispec_packed<1024>(plan, g, L, shell_bins, mas_order, data, st);
  }
  if (r) return r;
  return bispec_outputs(B, part, L.groups, E, shell_bins, n_shells, N, box_size, pk_out, bk_out, qk_out, nmodes_out,
                        st);
}

}  // namespace
}  // namespace gbp

using namespace gbp;

extern "C" int gbp_bispec_workspace_size(gbp_fft_plan plan, gbp_bins B, size_t* bytes) {
  if (!plan || !B || !bytes || plan->n != B->N || plan->grids != 1) return GBP_ERR_INVALID;
  BpLayout Lp;
  if (bp_layout(plan, B, Lp) == GBP_OK) {
    *bytes = Lp.total_ws;
    return GBP_OK;
  }
  BkLayout L;
  const int st = bk_layout(plan, B, L);
  if (st) return st;
  *bytes = L.total_ws;
  return GBP_OK;
}

extern "C" int gbp_bispec(gbp_fft_plan plan, const float* delta, void* spectrum, gbp_bins B, int mas_order,
                          const int32_t* shell_bins, int n_shells, double box_size, double* pk_out, double* bk_out,
                          double* qk_out, long long* nmodes_out, void* workspace, size_t ws_bytes,
                          gbp_stream_t stream_) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  if (!plan || !delta || !spectrum || !B || !shell_bins || !pk_out || !(box_size > 0.0)) return GBP_ERR_INVALID;
  if (plan->n != B->N || plan->grids != 1 || mas_order < 0 || mas_order > 8 || n_shells < 2) return GBP_ERR_INVALID;
  if (n_shells > 2 && (!bk_out || !qk_out)) return GBP_ERR_INVALID;
  BpLayout Lp;
  if (bp_layout(plan, B, Lp) == GBP_OK)
    return bispec_packed(plan, delta, spectrum, B, mas_order, shell_bins, n_shells, box_size, pk_out, bk_out, qk_out,
                         nmodes_out, workspace, ws_bytes, Lp, st);
  BkLayout L;
  int r = bk_layout(plan, B, L);
  if (r) return r;
  if (!workspace || ws_bytes < L.total_ws) return GBP_ERR_WORKSPACE;
  const int N = plan->n, P = plan->pitch;
  const long long M = (long long)N * N * N, T = (long long)N * N * L.Pc;
  Carver cv(workspace);
  float2* A = cv.take<float2>(L.A / sizeof(float2));
  float* R = cv.take<float>(L.R / sizeof(float));
  float2* part = cv.take<float2>(L.part / sizeof(float2));
  double* E = cv.take<double>(L.E / sizeof(double));
  void* cws = cv.take<char>(L.cws);
  // 1. forward transform of the contrast
  r = gbp_fft_r2c(plan, delta, spectrum, cws, L.cws, stream_);
  if (r) return r;
  // 2. the first two shells' masked spectra and masks
  {
    GBP_TRACE("bispec_fill", st);
    bispec_fill_kernel<<<(unsigned)((T + 255) / 256), 256, 0, st>>>(static_cast<const float2*>(spectrum), P, A,
                                                                     L.Pc, N, B->d_thr, B->nbe, shell_bins,
                                                                     B->d_inv_sinc2, mas_order);
    GBP_LAUNCH_CHECK();
  }
  // 3. their fields
  {
    GBP_TRACE("bispec_c2r", st);
    r = c2r_exec(N, L.Pc, 4, A, R, cws, st);
    if (r) return r;
  }
  // 4. delta_1 delta_2 and I_1 I_2
  int dev = 0, sms = 0;
  GBP_CUDA_TRY(cudaGetDevice(&dev));
  GBP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  {
    GBP_TRACE("bispec_products", st);
    const long long work = (M & 3) == 0 ? M / 4 : M;
    const int grid = (int)std::max(1LL, std::min((long long)sms * 8, (work + 255) / 256));
    bispec_products_kernel<<<grid, 256, 0, st>>>(R, M);
    GBP_LAUNCH_CHECK();
  }
  // 5. their spectra (the plan's transform), over the consumed half spectra
  float2* sD = A;
  float2* sJ = A + (long long)N * N * P;
  r = gbp_fft_r2c(plan, R, sD, cws, L.cws, stream_);
  if (r) return r;
  r = gbp_fft_r2c(plan, R + M, sJ, cws, L.cws, stream_);
  if (r) return r;
  // 6. one pass over the spectrum into elementary bins
  PowGeom g = bk_geom(plan, B, spectrum, part);
  g.total = L.total;
  g.chunk = L.chunk;
  g.warps = L.warps;
  g.groups = L.C;
  int per_sm = 0;
  GBP_CUDA_TRY(cudaFuncSetAttribute(bispec_bin_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem));
  GBP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, bispec_bin_kernel, L.warps * 32, L.smem));
  {
    GBP_TRACE("bispec_bins", st);
    const int grid = std::max(1, std::min(L.C, sms * std::max(per_sm, 1)));
    bispec_bin_kernel<<<grid, L.warps * 32, L.smem, st>>>(g, sD, sJ, mas_order);
    GBP_LAUNCH_CHECK();
  }
  return bispec_outputs(B, part, L.C, E, shell_bins, n_shells, N, box_size, pk_out, bk_out, qk_out, nmodes_out, st);
}
