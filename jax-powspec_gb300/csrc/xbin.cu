// The x pass of the 3-D FFT fused with the binning.
//
// After the z and y passes (fft.cu) the spectrum buffer holds the packed
// field Z transformed over z and y: slab 0 at kz, slab 1 at -kz; the
// remaining 1-D transforms run along x, whose rows lie N*P complex apart.
// Instead of writing them back and reading them again for the binning, one
// CTA takes a work item = one ky row and a block of 8 adjacent kz columns of
// slab 0, and row -ky of the same block of slab 1:
//
//   1. loads the item's 2 x NX x 8 complex values (16-byte loads, 64
//      contiguous bytes per x row) into shared memory,
//   2. transforms the 16 columns along x (NX = N points for an interlaced
//      pair, N/2 for one grid) with radix-8 Stockham stages (fft_core.cuh);
//      the last stage writes the result column-major with an XOR swizzle, so
//      the binning reads it without bank conflicts,
//   3. bins the 8 x N modes.  With A = Z(k), B = conj Z(-k) the mode is
//          two grids:  F0 + phi F1,  F0 = (A + B)/2, F1 = -i (A - B)/2,
//                      phi = exp(i pi (kx + ky + kz) / N)  (times 1/2)
//          one grid:   E + w O, the same with w = exp(-2 pi i kx / N) and
//                      Z taken at kx mod N/2,
//      that is ((A + B) - i f (A - B)) / 2 with f = phi or w (the fields come
//      times 1/4 or 1/2, so the mode needs no factor).  The modes x and N - x
//      of a column (kx and -kx) share |k|, mu, the window and the bin, and the
//      four values they need, so they are summed first and looked up once; a
//      warp walks one column over half of the |kx| range
//      (or all of it; x = N/2 alone is added after the last pair), so bins
//      are monotone along the walk.  A lane owns consecutive pairs; runs of
//      equal bin are summed in-lane, joined across lanes by one warp
//      segmented scan, and each run is added once to the warp's float32 bins
//      (distinct bins within a step: no atomics).
//
// Only items with a mode inside the last k edge are listed by the bin plan
// (gbp_bins_create): edges up to k_Nyquist leave out a fifth of them.  Two
// grids at 512^3: 0.688 -> 0.552 ms, 0.526 with loads that keep their lines in
// L2, 0.438 with interleaved planes (0.86 GB read: 2.0 TB/s; 1024^3 5.16 ->
// 4.34 ms, 256^3 0.074 -> 0.063); one grid (half the points per column, a warp
// per column): 0.545 -> 0.362, 0.330, 0.285 ms at 512^3.  Bound by barriers,
// shared-memory wavefronts (half the pipe) and issue (0.4 of the slots).  Items
// of 4 columns (half the threads per barrier) took 0.543 ms, for their 32-byte
// rows, before the interleaving.
//
// The mode arithmetic (window deconvolution, interlacing average, |delta|^2,
// mu^2 and mu^4 moments, DC removal) and the bin lookup are those of
// power.cu.  CTA g walks work group g (items g, g + groups, ...); each
// group folds its warps' bins in a fixed order into
// a float-float partial, and power_reduce_kernel folds the partials into
// doubles, so results are bitwise reproducible on every device.  The full
// spectrum never returns to HBM: the pipeline reads 8 bytes per mode here
// instead of writing and reading them three more times.
#include <algorithm>

#include "xpass.cuh"

namespace gbp {
namespace {

constexpr int XB_BINS = 8;                   // per-warp bin arrays; warps w and w + 8 share one

// Moments and bins of one warp step of mode pairs: lane pairs p0 .. p0 + MS - 1
// of a column (a_col at (ky, kz), b_col at (-ky, -kz)), pair p = the modes
// kx = p and -p, whose |k|, mu, window and bin agree; p = 0 is one mode.
// eyz: the ky and kz part of the phase (two grids).
template <int N, int NV, bool INTER, int MS>
__device__ __forceinline__ void xbin_pairs(const PowGeom& g, const Smem& t, const float* c2x, const float2* fx,
                                           const float2* a_col, const float2* b_col, int p0, int kyz2, float cyz,
                                           float fz2, float2 eyz, float (&P)[MS][NV], int (&bin)[MS]) {
  using L = XLayout<N, INTER>;
#pragma unroll
  for (int j = 0; j < MS; ++j) {
    const int p = p0 + j;
    const int sp = xswz<L::M2>(p), sm = xswz<L::M2>((L::NX - p) & (L::NX - 1));
    const float2 e = fx[sp];
    float fr = e.x, fi = e.y, mr = e.x, mi = -e.y;           // f of kx = p and of kx = -p
    if (INTER) {
      const float ar = e.x * eyz.x, ai = e.x * eyz.y, br = e.y * eyz.y, bi = e.y * eyz.x;
      fr = ar - br;
      fi = ai + bi;
      mr = ar + br;
      mi = ai - bi;
    }
    const float2 ap = a_col[sp], am = a_col[sm], bp = b_col[sp], bm = b_col[sm];
    const float2 u = unpack_mode(ap, bm, fr, fi), v = unpack_mode(am, bp, mr, mi);
    const int k2 = p * p + kyz2;
    float pw = u.x * u.x + u.y * u.y;
    if (g.zero_dc && k2 == 0) pw = 0.0f;
    if (p > 0) pw += v.x * v.x + v.y * v.y;
    const float w = pw * (cyz * c2x[sp]);
    P[j][0] = w;
    if (NV > 1) {
      const float mu2 = k2 > 0 ? __fdividef(fz2, (float)k2) : 0.0f;
      P[j][1] = w * mu2;
      if (NV > 2) P[j][2] = P[j][1] * mu2;
    }
    bin[j] = bin_of(g, t, k2);
  }
}

// The mode kx = N/2 (its own mirror) of one column, added to the warp's bins
// by one lane.  Out of line: it runs once per column and only for bins
// beyond k_Nyq, and inlined it would cost the binning registers.
template <int N, int NV, bool INTER>
__device__ __noinline__ void add_nyquist_x(const PowGeom& g, const Smem& t, const float2* a_col, const float2* b_col,
                                           int kyz2, float cyz, float fz2, float2 eyz, float* wb) {
  using L = XLayout<N, INTER>;
  constexpr int H = N / 2;
  const int sp = xswz<L::M2>(H & (L::NX - 1));
  float fr = -1.0f, fi = 0.0f;                               // w^(N/2)
  if (INTER) {
    const float2 e = t.eph[H];
    fr = e.x * eyz.x - e.y * eyz.y;
    fi = e.x * eyz.y + e.y * eyz.x;
  }
  const float2 u = unpack_mode(a_col[sp], b_col[sp], fr, fi);
  const int k2 = H * H + kyz2;
  float P[NV];
  P[0] = (u.x * u.x + u.y * u.y) * (cyz * t.c2[H]);
  if (NV > 1) {
    const float mu2 = __fdividef(fz2, (float)k2);
    P[1] = P[0] * mu2;
    if (NV > 2) P[2] = P[1] * mu2;
  }
  const int bin = bin_of(g, t, k2);
  if (bin >= 0) bin_add<NV>(wb, g.nbe, bin, P);
}

// Bin the 8 columns of one item (transposed layout in s).  HALVES = 2: warp
// w takes column w / 2 and half w % 2 of the |kx| range; warps w and w + 8
// share bin array w % 8 and flush in two phases separated by barriers.
// HALVES = 1: warp w takes column w.  No barrier follows the last step: the
// caller's next barrier (the next item's first FFT stage, or the fold)
// orders the last flushes and reads of s.
template <int N, int NV, bool INTER>
__device__ __forceinline__ void xbin_item(const PowGeom& g, const Smem& t, const float* c2x, const float2* fx,
                                          const float2* s, int warp, int lane, int y, int kb) {
  using L = XLayout<N, INTER>;
  constexpr int H = N / 2, TST = L::TST, HALVES = L::HALVES, M2 = L::M2, MS2 = L::MS2;
  const int c = warp / HALVES, h = warp % HALVES;
  const int kz = kb * XB_C + c;
  const bool active = kz <= H;                              // else row padding
  const int kzc = active ? kz : 0;
  const int ky = signed_k(y, N);
  const int ay = ky < 0 ? -ky : ky;
  float2 eyz = make_float2(1.f, 0.f);
  if (INTER) {
    float2 ey = t.eph[ay];
    if (ky < 0) ey.y = -ey.y;
    const float2 ez = t.eph[kzc];
    eyz = make_float2(ey.x * ez.x - ey.y * ez.y, ey.x * ez.y + ey.y * ez.x);
  }
  const float cyz = t.c2[ay] * t.c2[kzc];
  const int kyz2 = ky * ky + kzc * kzc;
  const float fz2 = (float)(kzc * kzc);
  const float2* a_col = s + c * TST;
  const float2* b_col = s + (XB_C + c) * TST;
  float* wb = t.wbase + (warp & (XB_BINS - 1)) * NV * g.nbe;
#pragma unroll 1
  for (int s0 = 0; s0 < M2; s0 += MS2) {
    float P[MS2][NV];
    int bin[MS2];
    if (active)
      xbin_pairs<N, NV, INTER, MS2>(g, t, c2x, fx, a_col, b_col, h * (H / HALVES) + lane * M2 + s0, kyz2, cyz, fz2,
                                    eyz, P, bin);
    auto flush = [&]() {
      flush_runs<MS2, NV>(P, bin, lane, wb, g.nbe);
      // |kx| = N/2 reaches a bin only when the last edge lies beyond k_Nyq
      if (h == HALVES - 1 && s0 + MS2 >= M2 && (H * H + kyz2 <= g.tu)) {
        if (lane == 0) add_nyquist_x<N, NV, INTER>(g, t, a_col, b_col, kyz2, cyz, fz2, eyz, wb);
        __syncwarp();
      }
    };
    if constexpr (HALVES == 1) {
      if (active) flush();
    } else {
      if (warp < XB_BINS && active) flush();
      __syncthreads();
      if (warp >= XB_BINS && active) flush();
      if (s0 + MS2 < M2) __syncthreads();   // after the last step, the next item's (or the fold's) barrier follows
    }
  }
}

template <int N, int NV, bool INTER>
__global__ void __launch_bounds__(XLayout<N, INTER>::NT,
                                  N >= 1024 && INTER ? 1 : 1024 / XLayout<N, INTER>::NT)
xbin_kernel(PowGeom g) {
  pdl_wait();
  using L = XLayout<N, INTER>;
  constexpr int NT = L::NT;
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = reinterpret_cast<float2*>(smem);
  float2* fx = reinterpret_cast<float2*>(smem + L::data_bytes());
  float* c2x = reinterpret_cast<float*>(fx + N / 2);
  const Smem t = load_tables<NV, INTER>(g, smem + L::data_bytes() + L::xtab_bytes());
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int p = tid; p < N / 2; p += NT) {                   // per-|kx| tables (load_tables ended with a barrier)
    fx[xswz<L::M2>(p)] = INTER ? t.eph[p] : g.tw[p];        // exp(i pi p / N), exp(-2 pi i p / N)
    c2x[xswz<L::M2>(p)] = t.c2[p];
  }
  __syncthreads();
  for (int grp = blockIdx.x; grp < g.groups; grp += gridDim.x) {
    for (int it = grp; it < g.items; it += g.groups) {
      const int code = __ldg(g.item_list + it), y = code / XITEM_KB, kb = code % XITEM_KB;
      // from 512^3 up the first stage loads the item from HBM while the previous item's last warps
      // still bin it, and waits for them before it writes the shared buffer (smaller meshes: the
      // registers the early loads hold would spill; they end the binning with a barrier instead)
      x_forward<N, INTER, XB_EARLY<N>>(s, g.s0, y, kb, g.twx, tid);
      xbin_item<N, NV, INTER>(g, t, c2x, fx, s, warp, lane, y, kb);
      if constexpr (!XB_EARLY<N>) __syncthreads();
    }
    cta_fold<NV>(g, t, grp);
  }
}

// Work groups: a pure function of the items, so the summation order is the
// same on every device.
int xbin_groups(int items) { return std::max(1, std::min(items, 1216)); }

struct XbLayout {
  int NV, items, groups;
  size_t smem, ws;
};

int xbin_layout(const gbp_bins_s* B, int G, int ells, XbLayout& L) {
  const int N = B->N;
  L.NV = (ells & GBP_ELL4) ? 3 : ((ells & GBP_ELL2) ? 2 : 1);
  L.items = B->n_xitems;
  L.groups = xbin_groups(L.items);
  size_t data = 0;
#define GBP_DATA(NN) \
  case NN: data = G == 2 ? XLayout<NN, true>::data_bytes() : XLayout<NN, false>::data_bytes(); break
  switch (N) {
    GBP_DATA(64);
    GBP_DATA(128);
    GBP_DATA(256);
    GBP_DATA(512);
    GBP_DATA(1024);
    default: return GBP_ERR_UNSUPPORTED;
  }
#undef GBP_DATA
  L.smem = data + (size_t)(N / 2) * 12 + smem_plan(N, B->nbe, B->lut_n, XB_BINS, L.NV).total;
  if (L.smem > 227 * 1024) return GBP_ERR_UNSUPPORTED;
  L.ws = align256((size_t)L.groups * L.NV * B->nbe * sizeof(float2));
  return GBP_OK;
}

template <int N, int NV, bool INTER>
int launch_xbin(const PowGeom& g, size_t smem, cudaStream_t st) {
  auto k = xbin_kernel<N, NV, INTER>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // one CTA per work group (not a persistent grid): CTAs end every ~14 items, so the block
  // scheduler can start a higher-priority stream's kernels (small serving requests) in between;
  // as fast as the persistent grid at 512^3 (0.775 against 0.781 ms)
  const int grid = std::max(1, g.groups);
  GBP_TRACE("fft_x_bins", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3(grid), dim3(XLayout<N, INTER>::NT), smem, st, g));
  return GBP_OK;
}

template <int N>
int dispatch_xbin(const PowGeom& g, int NV, bool inter, size_t smem, cudaStream_t st) {
  if (inter) {
    if (NV == 3) return launch_xbin<N, 3, true>(g, smem, st);
    if (NV == 2) return launch_xbin<N, 2, true>(g, smem, st);
    return launch_xbin<N, 1, true>(g, smem, st);
  }
  if (NV == 3) return launch_xbin<N, 3, false>(g, smem, st);
  if (NV == 2) return launch_xbin<N, 2, false>(g, smem, st);
  return launch_xbin<N, 1, false>(g, smem, st);
}

}  // namespace
}  // namespace gbp

namespace gbp {

int xbin_power_workspace(gbp_fft_plan plan, gbp_bins B, int ells, size_t* bytes) {
  if (!plan || !B || !bytes || plan->n != B->N) return GBP_ERR_INVALID;
  if (!plan->own || (plan->grids != 1 && plan->grids != 2)) return GBP_ERR_UNSUPPORTED;
  XbLayout L;
  const int st = xbin_layout(B, plan->grids, ells, L);
  if (st) return st;
  *bytes = L.ws;
  return GBP_OK;
}

int xbin_power(gbp_fft_plan plan, float2* spec, gbp_bins B, int mas_order, int ells, const double* mass,
               double* sums_out, long long* nmodes_out, double* ksum_out, void* workspace, size_t ws_bytes,
               cudaStream_t st, const StatsFold& stats) {
  if (!plan || !spec || !B || !sums_out || !nmodes_out) return GBP_ERR_INVALID;
  if (plan->n != B->N) return GBP_ERR_INVALID;
  if (!plan->own || (plan->grids != 1 && plan->grids != 2)) return GBP_ERR_UNSUPPORTED;
  if (mas_order < 0 || mas_order > 8) return GBP_ERR_INVALID;
  if ((ells & (GBP_ELL0 | GBP_ELL2 | GBP_ELL4)) == 0 || (ells & ~15)) return GBP_ERR_INVALID;
  if ((ells & GBP_KSUM) && !ksum_out) return GBP_ERR_INVALID;
  if ((reinterpret_cast<uintptr_t>(spec) & 15u) != 0) return GBP_ERR_INVALID;
  XbLayout L;
  int r = xbin_layout(B, plan->grids, ells, L);
  if (r) return r;
  if (!workspace || ws_bytes < L.ws) return GBP_ERR_WORKSPACE;
  const int N = B->N, G = plan->grids;
  PowGeom g{};
  g.s0 = spec;
  g.N = N;
  g.Lz = N / 2 + 1;
  g.Lzs = plan->pitch;
  g.nb = B->nb;
  g.nbe = B->nbe;
  g.tu = B->last_closed;
  g.lut_shift = B->lut_shift;
  g.lut_n = B->lut_n;
  g.mas_order = mas_order;
  g.thr = B->d_thr;
  g.lut = B->d_lut;
  g.inv_sinc2 = B->d_inv_sinc2;
  g.eph = B->d_eph;
  g.zero_dc = mass != nullptr;
  g.part_ff = static_cast<float2*>(workspace);
  g.warps = XB_BINS;
  g.groups = L.groups;
  g.tw = plan->tw;
  g.twx = plan->twx;
  g.items = L.items;
  g.item_list = B->d_xitems;
  switch (N) {
    case 64: r = dispatch_xbin<64>(g, L.NV, G == 2, L.smem, st); break;
    case 128: r = dispatch_xbin<128>(g, L.NV, G == 2, L.smem, st); break;
    case 256: r = dispatch_xbin<256>(g, L.NV, G == 2, L.smem, st); break;
    case 512: r = dispatch_xbin<512>(g, L.NV, G == 2, L.smem, st); break;
    case 1024: r = dispatch_xbin<1024>(g, L.NV, G == 2, L.smem, st); break;
    default: r = GBP_ERR_UNSUPPORTED;
  }
  if (r) return r;
  GBP_TRACE("power_reduce", st);
  GBP_CUDA_TRY(launch_pdl(power_reduce_kernel, dim3(B->nb + (stats.out ? 1 : 0)), dim3(FOLD_THREADS), 0, st,
                          static_cast<const float2*>(g.part_ff), L.groups, L.NV, B->nb, B->nbe,
                          static_cast<const long long*>(B->d_nmodes), static_cast<const double*>(B->d_ksum), sums_out,
                          nmodes_out, (ells & GBP_KSUM) ? ksum_out : nullptr, stats));
  return GBP_OK;
}

}  // namespace gbp

using namespace gbp;

extern "C" int gbp_fft_power_workspace_size(gbp_fft_plan plan, gbp_bins B, int ells, size_t* bytes) {
  return xbin_power_workspace(plan, B, ells, bytes);
}

extern "C" int gbp_fft_power(gbp_fft_plan plan, const float* mesh, void* spectrum, gbp_bins B, int mas_order,
                             int ells, const double* mass, double* sums_out, long long* nmodes_out, double* ksum_out,
                             void* workspace, size_t ws_bytes, gbp_stream_t stream_) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  if (!plan || !mesh || !spectrum || !B || !sums_out || !nmodes_out) return GBP_ERR_INVALID;
  if (plan->n != B->N) return GBP_ERR_INVALID;
  if (!plan->own || (plan->grids != 1 && plan->grids != 2)) return GBP_ERR_UNSUPPORTED;
  if (((reinterpret_cast<uintptr_t>(mesh) | reinterpret_cast<uintptr_t>(spectrum)) & 15u) != 0) return GBP_ERR_INVALID;
  size_t need = 0;
  int r = xbin_power_workspace(plan, B, ells, &need);
  if (r) return r;
  if (!workspace || ws_bytes < need) return GBP_ERR_WORKSPACE;
  float2* spec = static_cast<float2*>(spectrum);
  r = own_fft_z_packed(B->N, plan->grids, mesh, spec, B->kz_cols, plan->tw, st);
  if (r) return r;
  r = own_fft_y_packed(B->N, plan->grids, spec, B->kz_cols, B->last_closed, plan->tw, st);
  if (r) return r;
  return xbin_power(plan, spec, B, mas_order, ells, mass, sums_out, nmodes_out, ksum_out, workspace, ws_bytes, st,
                    StatsFold{});
}
