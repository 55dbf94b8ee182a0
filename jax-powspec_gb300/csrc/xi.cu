// Two-point correlation multipoles xi_l(r) from the same |delta_k|^2 as P_l(k)
// (src/correlations.py:120-187 xi_vec, :641-712 compute_2pt_correlations):
//
//   1. forward R2C of the density contrast (the plan's transform),
//   2. pk_field_kernel: |delta_k|^2 (sinc)^(-2p) per axis, in place, as a
//      complex field with zero imaginary part,
//   3. inverse C2R (cuFFT, unnormalised: the field holds N^3 xi(r)),
//   4. xi_bin_kernel: separation shells on the full grid (signed offsets on
//      all three axes; integer r^2 against the bin plan's thresholds, the
//      jnp.histogram rule), moments sum xi, xi mu^2, xi mu^4 and the cell
//      count; runs along z are summed by warp segmented scans and flushed
//      half-pencil by half-pencil into per-warp float32 bins, folded in
//      float-float per work group and in double at the end (deterministic),
//   5. xi_reduce_kernel: Legendre sums and counts.
//
// For the library's transform sizes gbp_xi_shells does the same without the
// field: |delta_k|^2 is real and even, so xi(r) = xi(-r) and only the x planes
// 0 .. N/2 that hold a shell are formed.  The x pass of the packed transform
// (xpass.cuh) forms |delta_k|^2 W^2 of an item in shared memory and transforms
// it back along x in the same kernel, storing the x planes within the last
// edge; the y pass stores the rows within it; the z pass bins its pencils in
// shared memory, z and -z together, with weight 2 for 0 < x < N/2.
// 256^3, r < 0.2 L: 0.404 -> 0.157 ms of kernels (z 0.035, y 0.026, x 0.064,
// y of 52 planes 0.012, z + bins 0.017; the field path's C2R alone took 0.098
// and its binning 0.144).
//
// mu = r_z / r; at r = 0 it is NaN (xi_vec divides 0 by 0) or 0
// (compute_2pt_correlations guards it), selected by the caller.
#include <cufft.h>
#include <math.h>

#include <algorithm>

#include "xpass.cuh"

namespace gbp {
namespace {

constexpr int XI_NV = 4;      // sum xi, xi mu^2, xi mu^4, count

__global__ void pk_field_kernel(float2* spec, int N, int P, const float* __restrict__ inv_sinc2, int mas_order) {
  const long long total = (long long)N * N * P;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int kz = (int)(i % P);
  if (kz > N / 2) return;                         // row padding: never read by the C2R
  const int iy = (int)((i / P) % N), ix = (int)(i / ((long long)P * N));
  const int ax = abs(signed_k(ix, N)), ay = abs(signed_k(iy, N));
  float w = 1.0f;
  for (int p = 0; p < mas_order; ++p) w *= inv_sinc2[ax] * inv_sinc2[ay] * inv_sinc2[kz];
  const float2 v = spec[i];
  spec[i] = make_float2((v.x * v.x + v.y * v.y) * w, 0.0f);
}

// One warp step over 32 consecutive cells of the flat [N][N][N] field.
__device__ __forceinline__ void xi_step(const PowGeom& g, const Smem& t, const float* __restrict__ field, float* wb,
                                        int lane, long long f, long long end, int nan_origin) {
  const int N = g.N;
  const bool valid = f < end;
  float v[XI_NV] = {0.f, 0.f, 0.f, 0.f};
  int bin = -1;
  const int z = (int)(f % N);
  const long long pen = f / N;
  const int hp = (int)(pen * 2 + (z > N / 2 ? 1 : 0));       // half-pencil: |r_z| is monotone inside it
  if (valid) {
    const int y = (int)(pen % N), x = (int)(pen / N);
    const int rx = signed_k(x, N), ry = signed_k(y, N), rz = signed_k(z, N);
    const int r2 = rx * rx + ry * ry + rz * rz;
    bin = bin_of(g, t, r2);
    const float xi = field[f];
    float mu2;
    if (r2 > 0) mu2 = __fdividef((float)(rz * rz), (float)r2);
    else mu2 = nan_origin ? __int_as_float(0x7fc00000) : 0.0f;
    v[0] = xi;
    v[1] = xi * mu2;
    v[2] = v[1] * mu2;
    v[3] = 1.0f;
  }
  const int bprev = __shfl_up_sync(0xffffffffu, bin, 1);
  const int hprev = __shfl_up_sync(0xffffffffu, hp, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || bin != bprev || hp != hprev);
  seg_scan<XI_NV>(v, heads, lane);
  const bool segend = (lane == 31) || ((heads >> (lane + 1)) & 1u);
  // runs of different half-pencils in one step may share a bin: flush phase by phase
  const int rel = hp - __shfl_sync(0xffffffffu, hp, 0);
  const int nph = __reduce_max_sync(0xffffffffu, valid ? rel : 0) + 1;
  for (int ph = 0; ph < nph; ++ph) {
    if (segend && bin >= 0 && rel == ph) bin_add<XI_NV>(wb, g.nbe, bin, v);
    __syncwarp();
  }
}

__global__ void __launch_bounds__(POW_WARPS * 32, 4)
xi_bin_kernel(PowGeom g, const float* __restrict__ field, int nan_origin) {
  extern __shared__ __align__(16) unsigned char smem[];
  const Smem s = load_tables<XI_NV, false>(g, smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* wb = s.wbase + warp * XI_NV * g.nbe;
  for (int grp = blockIdx.x; grp < g.groups; grp += gridDim.x) {
    const long long beg = ((long long)grp * g.warps + warp) * g.chunk;
    const long long end = min(beg + g.chunk, g.total);
    for (long long f = beg + lane; f - lane < end; f += 32) xi_step(g, s, field, wb, lane, f, end, nan_origin);
    cta_fold<XI_NV>(g, s, grp);
  }
}

// One block per bin: the group partials folded in a fixed order (fold_bin),
// then the Legendre sums and the cell count.
__global__ void __launch_bounds__(FOLD_THREADS)
xi_reduce_kernel(const float2* __restrict__ part_ff, int C, int nb, int nbe, double* sums_out,
                 long long* counts_out) {
  const int b = blockIdx.x;
  if (b >= nb) return;                         // uniform over the block
  double m[XI_NV] = {0.0, 0.0, 0.0, 0.0};
  if (b < nbe) fold_bin<XI_NV>(part_ff, C, XI_NV, nbe, b, m);
  if (threadIdx.x == 0) {
    sums_out[b * 3 + 0] = m[0];
    sums_out[b * 3 + 1] = 1.5 * m[1] - 0.5 * m[0];
    sums_out[b * 3 + 2] = (35.0 * m[2] - 30.0 * m[1] + 3.0 * m[0]) * 0.125;
    counts_out[b] = (long long)llrint(m[3]);
  }
}

// Items (y, kb) of the packed transform: x pass, power of the 8 columns at
// (ky, kz), transform of the N powers (real; the columns at (ky, kz) and
// (-ky, -kz) mirror each other) along x, x planes 0 .. xmax stored to out
// [xmax + 1][N][P].
template <int N>
__global__ void __launch_bounds__(XLayout<N, false>::NT, 1024 / XLayout<N, false>::NT)
xi_x_kernel(PowGeom g, float2* __restrict__ out, int xmax) {
  pdl_wait();
  using L = XLayout<N, false>;
  constexpr int P = N / 2 + 8, TST = L::TST, NX = L::NX, NT = L::NT, H = N / 2, PW = N + 4;
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = reinterpret_cast<float2*>(smem);
  float* pw = reinterpret_cast<float*>(smem + L::data_bytes());            // [8][PW]
  const Smem t = load_tables<1, false>(g, smem + L::data_bytes() + (size_t)XB_C * PW * sizeof(float));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int it = blockIdx.x; it < g.items; it += gridDim.x) {
    const int y = it / (P / 8), kb = it - y * (P / 8);
    x_forward<N, false, false>(s, g.s0, y, kb, g.twx, tid);
    const int c = warp / L::HALVES, kz = kb * XB_C + c;
    const int ky = signed_k(y, N), ay = ky < 0 ? -ky : ky;
    const float cyz = kz <= H ? t.c2[ay] * t.c2[kz] : 0.0f;
    const float2* a = s + c * TST;
    const float2* b = s + (XB_C + c) * TST;
    for (int p = lane + 32 * (warp % L::HALVES); p <= H; p += 32 * L::HALVES) {
      const int sp = xswz<L::M2>(p & (NX - 1)), sm = xswz<L::M2>((NX - p) & (NX - 1));
      const float2 w = __ldg(g.tw + p);
      const float2 u = unpack_mode(a[sp], b[sm], w.x, w.y), v = unpack_mode(a[sm], b[sp], w.x, -w.y);
      const float cw = cyz * t.c2[p];
      pw[c * PW + p] = kz <= H ? (u.x * u.x + u.y * u.y) * cw : 0.0f;
      if (p > 0 && p < H) pw[c * PW + N - p] = kz <= H ? (v.x * v.x + v.y * v.y) * cw : 0.0f;
    }
    __syncthreads();
    auto gin = [pw](int j, int cp) {
      return make_float4(pw[2 * cp * PW + j], 0.0f, pw[(2 * cp + 1) * PW + j], 0.0f);
    };
    float2* dst = out + (long long)y * P + kb * XB_C;
    auto gout = [dst, xmax](int x, int cp, float4 v) {
      if (x <= xmax) __stcs(reinterpret_cast<float4*>(dst + (long long)x * N * P) + cp, v);
    };
    fft::col_fft<N, 1, NT, false>(s, gin, gout, g.tw, tid);
    __syncthreads();
  }
}

// z pass and binning.  An item is 2 PAIRS rows y of one x plane (two real
// pencils per complex column: h(-kz) = conj h(kz)); after the transform a warp
// walks one pencil, z and -z together, |z| ascending.
template <int N, int PAIRS>
__global__ void __launch_bounds__(PAIRS * N / 16)
xi_z_kernel(PowGeom g, const float2* __restrict__ h, int chunks, int nan_origin) {
  pdl_wait();
  constexpr int NT = PAIRS * N / 16, CP = PAIRS / 2, P = N / 2 + 8, H = N / 2;
  extern __shared__ __align__(16) unsigned char smem[];
  float4* s4 = reinterpret_cast<float4*>(smem);                            // [CP][N] slots of two columns
  const Smem t = load_tables<XI_NV, false>(g, smem + (size_t)PAIRS * N * sizeof(float2));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* wb = t.wbase + warp * XI_NV * g.nbe;
  for (int grp = blockIdx.x; grp < g.groups; grp += gridDim.x) {
    for (int it = grp; it < g.items; it += g.groups) {
      const int x = it / chunks, m0 = (it - x * chunks) * 2 * PAIRS;
      const int y2 = g.tu - x * x;                                         // rows with y^2 <= y2
      int ym = min((int)sqrtf((float)max(y2, 0)), H);
      while (ym > 0 && ym * ym > y2) --ym;
      while (ym < H && (ym + 1) * (ym + 1) <= y2) ++ym;
      const int rows = y2 < 0 ? 0 : min(N, 2 * ym + 1);
      if (m0 >= rows) continue;                                            // uniform over the block
      auto row_y = [ym, rows](int m) { return m <= ym ? m : N - rows + m; };
      auto at = [&](int f, int kz) {                                       // h of pencil f of the item
        const int m = m0 + f;
        return m < rows ? __ldcg(h + ((long long)x * N + row_y(m)) * P + kz) : make_float2(0.f, 0.f);
      };
      auto gin = [&](int j, int cp) {                                      // columns 2cp, 2cp+1: pencils 4cp .. 4cp+3
        const int kz = j <= H ? j : N - j;
        float2 q[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          q[k] = at(4 * cp + k, kz);
          if (j > H) q[k].y = -q[k].y;
          if (kz == 0 || kz == H) q[k].y = 0.0f;                           // real up to round-off
        }
        return make_float4(q[0].x - q[1].y, q[0].y + q[1].x, q[2].x - q[3].y, q[2].y + q[3].x);
      };
      auto sin_ = [s4](int j, int cp) { return s4[cp * N + fft::zsw(j)]; };
      auto sout = [s4](int j, int cp, float4 v) { s4[cp * N + fft::zsw(j)] = v; };
      fft::run_stages2<N, CP, NT, true, false, true>(gin, sin_, sout, sout, g.tw, tid);
      const float* sf = reinterpret_cast<const float*>(s4);
      const float wx = (x == 0 || x == H) ? 1.0f : 2.0f;
      for (int f = warp; f < 2 * PAIRS && m0 + f < rows; f += NT / 32) {
        const float* col = sf + (size_t)(f >> 2) * N * 4 + (f & 3);
        const int ry = signed_k(row_y(m0 + f), N);
        const int rp2 = x * x + ry * ry;
        for (int z0 = 0; z0 <= H && rp2 + z0 * z0 <= g.tu; z0 += 32) {
          const int z = z0 + lane;
          float v[XI_NV] = {0.f, 0.f, 0.f, 0.f};
          int bin = -1;
          if (z <= H) {
            const int r2 = rp2 + z * z;
            bin = bin_of(g, t, r2);
            const bool single = z == 0 || z == H;
            float xi = col[fft::zsw(z) * 4];
            if (!single) xi += col[fft::zsw(N - z) * 4];
            xi *= wx;
            float mu2;
            if (r2 > 0) mu2 = __fdividef((float)(z * z), (float)r2);
            else mu2 = nan_origin ? __int_as_float(0x7fc00000) : 0.0f;
            v[0] = xi;
            v[1] = xi * mu2;
            v[2] = v[1] * mu2;
            v[3] = single ? wx : 2.0f * wx;
          }
          const int bprev = __shfl_up_sync(0xffffffffu, bin, 1);
          const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || bin != bprev);
          seg_scan<XI_NV>(v, heads, lane);
          const bool segend = (lane == 31) || ((heads >> (lane + 1)) & 1u);
          if (segend && bin >= 0) bin_add<XI_NV>(wb, g.nbe, bin, v);
          __syncwarp();
        }
      }
      __syncthreads();
    }
    cta_fold<XI_NV>(g, t, grp);
  }
}

struct XiShells {
  int xmax, chunks, items, groups;
  size_t smem_x, smem_z, h, part, total;
};

template <int N>
constexpr int xi_pairs() { return N >= 256 ? 8 : 32768 / (N * 8); }   // >= 128 threads

template <int N>
int xi_shells_layout_n(const gbp_bins_s* B, XiShells& L) {
  using XL = XLayout<N, false>;
  constexpr int PAIRS = xi_pairs<N>(), H = N / 2;
  L.xmax = -1;
  while (L.xmax < H && (long long)(L.xmax + 1) * (L.xmax + 1) <= (long long)B->last_closed) ++L.xmax;
  const int rows = std::min(N, 2 * L.xmax + 1);
  L.chunks = L.xmax < 0 ? 1 : (rows + 2 * PAIRS - 1) / (2 * PAIRS);
  L.items = (L.xmax + 1) * L.chunks;
  L.groups = std::max(1, std::min(L.items, 1216));
  L.smem_x = XL::data_bytes() + (size_t)XB_C * (N + 4) * sizeof(float) + smem_plan(N, B->nbe, B->lut_n, 0, 1).total;
  L.smem_z = (size_t)PAIRS * N * sizeof(float2) + smem_plan(N, B->nbe, B->lut_n, PAIRS * N / 512, XI_NV).total;
  if (L.smem_x > 227 * 1024 || L.smem_z > 227 * 1024) return GBP_ERR_UNSUPPORTED;
  L.h = align256((size_t)(L.xmax + 1) * N * (N / 2 + 8) * sizeof(float2));
  L.part = align256((size_t)L.groups * XI_NV * B->nbe * sizeof(float2));
  L.total = L.h + L.part;
  return GBP_OK;
}

int xi_shells_layout(const gbp_bins_s* B, XiShells& L) {
  switch (B->N) {
    case 64: return xi_shells_layout_n<64>(B, L);
    case 128: return xi_shells_layout_n<128>(B, L);
    case 256: return xi_shells_layout_n<256>(B, L);
    case 512: return xi_shells_layout_n<512>(B, L);
    case 1024: return xi_shells_layout_n<1024>(B, L);
    default: return GBP_ERR_UNSUPPORTED;
  }
}

template <int N>
int run_xi_shells(gbp_fft_plan plan, PowGeom g, const XiShells& L, float2* h, float2* part, int nan_origin,
                  cudaStream_t st) {
  using XL = XLayout<N, false>;
  constexpr int PAIRS = xi_pairs<N>(), P = N / 2 + 8;
  const float2* tw = plan->tw;
  if (L.xmax >= 0) {
    auto k = xi_x_kernel<N>;
    GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem_x));
    g.warps = 0;
    g.items = N * (P / 8);
    GBP_TRACE("xi_x", st);
    GBP_CUDA_TRY(launch_pdl(k, dim3(std::min(g.items, 1216)), dim3(XL::NT), L.smem_x, st, g, h, L.xmax));
  }
  const int r = own_fft_y_shells(N, h, L.xmax + 1, g.tu, tw, st);
  if (r) return r;
  auto k = xi_z_kernel<N, PAIRS>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem_z));
  g.warps = PAIRS * N / 512;
  g.items = L.items;
  g.groups = L.groups;
  g.part_ff = part;
  g.mas_order = 0;
  GBP_TRACE("xi_z_bins", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3(L.groups), dim3(PAIRS * N / 16), L.smem_z, st, g, static_cast<const float2*>(h),
                          L.chunks, nan_origin));
  return GBP_OK;
}

struct XiLayout {
  int warps, C;
  long long total, chunk;
  size_t smem, part, c2r_ws, total_ws;
};

int xi_layout(const gbp_bins_s* B, int P, size_t r2c_ws, XiLayout& L) {
  const int N = B->N;
  int w = POW_WARPS;
  while (w > 1 && smem_plan(N, B->nbe, B->lut_n, w, XI_NV).total > 200 * 1024) --w;
  L.smem = smem_plan(N, B->nbe, B->lut_n, w, XI_NV).total;
  if (L.smem > 200 * 1024) return GBP_ERR_UNSUPPORTED;
  L.warps = w;
  L.total = (long long)N * N * N;
  long long target = L.total / (8LL * 152 * 8);
  target = std::max(1024LL, std::min(16384LL, target));
  L.chunk = (target + 31) & ~31LL;
  const long long nw = (L.total + L.chunk - 1) / L.chunk;
  L.C = (int)((nw + w - 1) / w);
  L.part = align256((size_t)L.C * XI_NV * B->nbe * sizeof(float2));
  cufftHandle h;
  int st = c2r_plan(N, P, 1, &h, &L.c2r_ws);
  if (st) return st;
  if (r2c_ws > L.c2r_ws) L.c2r_ws = r2c_ws;          // one work area serves both transforms
  L.total_ws = L.part + align256(L.c2r_ws);
  return GBP_OK;
}

}  // namespace
}  // namespace gbp

using namespace gbp;

extern "C" int gbp_xi_workspace_size(gbp_fft_plan plan, gbp_bins B, size_t* bytes) {
  if (!plan || !B || !bytes || plan->n != B->N || plan->grids != 1) return GBP_ERR_INVALID;
  XiLayout L;
  const int st = xi_layout(B, plan->pitch, plan->ws, L);
  if (st) return st;
  *bytes = L.total_ws;
  return GBP_OK;
}

extern "C" int gbp_xi(gbp_fft_plan plan, const float* delta, void* spectrum, float* field, gbp_bins B, int mas_order,
                      int nan_mu_at_origin, double* sums_out, long long* counts_out, void* workspace,
                      size_t ws_bytes, gbp_stream_t stream_) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  if (!plan || !delta || !spectrum || !field || !B || !sums_out || !counts_out) return GBP_ERR_INVALID;
  if (plan->n != B->N || plan->grids != 1 || mas_order < 0 || mas_order > 8) return GBP_ERR_INVALID;
  XiLayout L;
  int r = xi_layout(B, plan->pitch, plan->ws, L);
  if (r) return r;
  if (!workspace || ws_bytes < L.total_ws) return GBP_ERR_WORKSPACE;
  const int N = B->N, P = plan->pitch;
  Carver cv(workspace);
  float2* part = cv.take<float2>(L.part / sizeof(float2));
  void* cws = cv.take<char>(L.c2r_ws);
  // 1. forward transform (library or cuFFT, as the plan says)
  r = gbp_fft_r2c(plan, delta, spectrum, cws, L.c2r_ws, stream_);
  if (r) return r;
  // 2. |delta_k|^2 W(k)^2
  float2* spec = static_cast<float2*>(spectrum);
  const long long total = (long long)N * N * P;
  {
    GBP_TRACE("xi_pk_field", st);
    pk_field_kernel<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(spec, N, P, B->d_inv_sinc2, mas_order);
    GBP_LAUNCH_CHECK();
  }
  // 3. inverse real transform (unnormalised)
  {
    GBP_TRACE("xi_c2r", st);
    r = c2r_exec(N, P, 1, spec, field, cws, st);
    if (r) return r;
  }
  // 4. separation shells
  PowGeom g{};
  g.N = N;
  g.total = L.total;
  g.chunk = L.chunk;
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
  g.warps = L.warps;
  g.groups = L.C;
  int dev = 0, sms = 0, per_sm = 0;
  GBP_CUDA_TRY(cudaGetDevice(&dev));
  GBP_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  GBP_CUDA_TRY(cudaFuncSetAttribute(xi_bin_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem));
  GBP_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, xi_bin_kernel, L.warps * 32, L.smem));
  const int grid = std::max(1, std::min(L.C, sms * std::max(per_sm, 1)));
  {
    GBP_TRACE("xi_bins", st);
    xi_bin_kernel<<<grid, L.warps * 32, L.smem, st>>>(g, field, nan_mu_at_origin ? 1 : 0);
    GBP_LAUNCH_CHECK();
  }
  {
    GBP_TRACE("xi_reduce", st);
    xi_reduce_kernel<<<B->nb, FOLD_THREADS, 0, st>>>(part, L.C, B->nb, B->nbe, sums_out, counts_out);
    GBP_LAUNCH_CHECK();
  }
  return GBP_OK;
}

extern "C" int gbp_xi_shells_workspace_size(gbp_fft_plan plan, gbp_bins B, size_t* bytes) {
  if (!plan || !B || !bytes || plan->n != B->N || plan->grids != 1) return GBP_ERR_INVALID;
  if (!plan->own) return GBP_ERR_UNSUPPORTED;
  XiShells L;
  const int st = xi_shells_layout(B, L);
  if (st) return st;
  *bytes = L.total;
  return GBP_OK;
}

extern "C" int gbp_xi_shells(gbp_fft_plan plan, const float* delta, void* spectrum, gbp_bins B, int mas_order,
                             int nan_mu_at_origin, double* sums_out, long long* counts_out, void* workspace,
                             size_t ws_bytes, gbp_stream_t stream_) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  if (!plan || !delta || !spectrum || !B || !sums_out || !counts_out) return GBP_ERR_INVALID;
  if (plan->n != B->N || plan->grids != 1 || mas_order < 0 || mas_order > 8) return GBP_ERR_INVALID;
  if (!plan->own) return GBP_ERR_UNSUPPORTED;
  if (((reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(spectrum)) & 15u) != 0) return GBP_ERR_INVALID;
  XiShells L;
  int r = xi_shells_layout(B, L);
  if (r) return r;
  if (!workspace || ws_bytes < L.total) return GBP_ERR_WORKSPACE;
  const int N = B->N, P = plan->pitch;
  Carver cv(workspace);
  float2* h = cv.take<float2>(L.h / sizeof(float2));
  float2* part = cv.take<float2>(L.part / sizeof(float2));
  float2* spec = static_cast<float2*>(spectrum);
  if (L.xmax >= 0) {
    r = own_fft_z_packed(N, 1, delta, spec, P, plan->tw, st);
    if (r) return r;
    r = own_fft_y_packed(N, 1, spec, P, 1 << 30, plan->tw, st);
    if (r) return r;
  }
  PowGeom g{};
  g.s0 = spec;
  g.N = N;
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
  g.tw = plan->tw;
  g.twx = plan->twx;
  switch (N) {
    case 64: r = run_xi_shells<64>(plan, g, L, h, part, nan_mu_at_origin ? 1 : 0, st); break;
    case 128: r = run_xi_shells<128>(plan, g, L, h, part, nan_mu_at_origin ? 1 : 0, st); break;
    case 256: r = run_xi_shells<256>(plan, g, L, h, part, nan_mu_at_origin ? 1 : 0, st); break;
    case 512: r = run_xi_shells<512>(plan, g, L, h, part, nan_mu_at_origin ? 1 : 0, st); break;
    case 1024: r = run_xi_shells<1024>(plan, g, L, h, part, nan_mu_at_origin ? 1 : 0, st); break;
    default: r = GBP_ERR_UNSUPPORTED;
  }
  if (r) return r;
  GBP_TRACE("xi_reduce", st);
  xi_reduce_kernel<<<B->nb, FOLD_THREADS, 0, st>>>(part, L.groups, B->nb, B->nbe, sums_out, counts_out);
  GBP_LAUNCH_CHECK();
  return GBP_OK;
}
