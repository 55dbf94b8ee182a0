// 3-D real-to-complex FFT of G meshes of side N (power of two, 64..1024) as
// three passes over HBM, each a batch of 1-D transforms staged in shared
// memory (fft_core.cuh):
//
//   z pass  real [G][N][N][N] -> complex [G][N][N][P], P = N/2 + 8: two real
//           z pencils are packed as one complex pencil (a + i b), transformed,
//           and split into their half spectra A, B (k = 0 .. N/2):
//             A[k] = (C[k] + conj C[N-k]) / 2,  B[k] = -i (C[k] - conj C[N-k]) / 2
//   y pass  in place, 8 adjacent kz columns x N rows per CTA; the first
//           stage reads HBM and the last writes it (fft_pass.cuh)
//   x pass  in place, same with rows N*P apart (the pipeline fuses it with
//           the binning instead: xbin.cu)
//
// The power spectrum needs no spectrum in that order, and takes the packed
// transform instead: one complex field c = a + i b of two real ones, whose
// spectrum Z carries both (A, B) = ((Z(k) + conj Z(-k)) / 2,
// -i (Z(k) - conj Z(-k)) / 2), is transformed along z, y and x without any
// split; the binning (xbin.cu) combines Z(k) and Z(-k) where it has both.
//
//   two grids   a, b = the two meshes of an interlaced pair; N x planes
//   one grid    a, b = the x planes 2x', 2x'+1 of the mesh; N/2 x' planes
//               (the last butterfly of the x transform, F(kx) = A + w^kx B)
//
// Layout [2][NX][N][P], NX = N (two grids) or N/2 (one): slab 0 holds Z at
// kz = 0 .. N/2, slab 1 holds Z at -kz, so both halves of a kz block are
// aligned and the y pass treats the slabs as two grids.  The split it saves
// cost the z pass a write and a read of the block in shared memory.  The x
// planes are interleaved four by four in blocks of 8 kz (fft::PackedRows): a
// block of one plane is half a 128-byte line, and the x pass, which reads one
// block of every plane for its row, finds four planes' blocks side by side.
// Columns and rows beyond the last k edge are not stored.
//
// The z rows are padded from N/2+1 to P = N/2+8 complex (64-byte multiples)
// so every 8-column block of the y and x passes is a whole number of 32-byte
// sectors; the padding is written as zeros by the z pass.  Same transform as
// cuFFT's R2C (forward, unnormalised) and numpy's rfftn.
#include <math.h>

#include <new>
#include <vector>

#include "fft_core.cuh"
#include "fft_pass.cuh"
#include "gbp_fft.h"
#include "gbp_internal.cuh"

namespace gbp {
namespace {

using fft::cadd;
using fft::cmi;
using fft::csub;
using fft::PACK_W;

__host__ __device__ constexpr int zpitch(int N) { return N / 2 + 8; }

// ---- z pass ---------------------------------------------------------------
// PAIRS complex columns (2*PAIRS real pencils) per CTA; a thread transforms
// two columns (four pencils) at once, NT = (PAIRS / 2) * N / 8.  Consecutive
// lanes take consecutive z, so the first stage's loads of each pencil are
// 128-byte coalesced.  Shared memory is column-major in 16-byte slots of two
// columns (fft_pass.cuh).  The last stage stays in shared memory, where each
// half spectrum needs C[k] and C[N-k] together.
using fft::zsw;

template <int N, int PAIRS>
__global__ void __launch_bounds__(PAIRS * N / 16)
fftz_kernel(const float* __restrict__ mesh, float2* __restrict__ out, long long npencils,
            const float2* __restrict__ tw) {
  pdl_wait();
  constexpr int NT = PAIRS * N / 16;
  constexpr int CP = PAIRS / 2;
  constexpr int P = zpitch(N);
  constexpr int H = N / 2;
  extern __shared__ __align__(16) float4 s4[];    // [CP][N] slots of two columns
  const int tid = threadIdx.x;
  const long long pen0 = (long long)blockIdx.x * 2 * PAIRS;
  const long long left = npencils - pen0;
  const int npen = left < 2 * PAIRS ? (int)left : 2 * PAIRS;
  const float* base = mesh + pen0 * N;

  auto gin = [base, npen](int j, int cp) {      // pencils 4cp .. 4cp+3 at z = j
    float v[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) v[f] = 4 * cp + f < npen ? __ldcg(base + (4 * cp + f) * N + j) : 0.0f;
    return make_float4(v[0], v[1], v[2], v[3]);
  };
  auto sin_ = [](int j, int cp) { return s4[cp * N + zsw(j)]; };
  auto sout = [](int j, int cp, float4 v) { s4[cp * N + zsw(j)] = v; };
  fft::run_stages2<N, CP, NT, true, false, true>(gin, sin_, sout, sout, tw, tid);

  // split the packed spectra and write both pencils' rows (padding -> 0); two k per thread and
  // 16-byte stores (rows are P = N/2 + 8 complex: 16-byte aligned)
  const float2* s2 = reinterpret_cast<const float2*>(s4);
  constexpr int P2 = P / 2;
  for (int idx = tid; idx < PAIRS * P2; idx += NT) {
    const int q = idx / P2, k0 = 2 * (idx - q * P2);
    if (2 * q >= npen) continue;
    const float2* col = s2 + (q >> 1) * N * 2 + (q & 1);
    float2 a[2], b[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + h;
      a[h] = b[h] = make_float2(0.f, 0.f);
      if (k <= H) {
        const float2 c = col[zsw(k) * 2];
        const float2 m = col[zsw((N - k) & (N - 1)) * 2];
        const float2 cm = make_float2(m.x, -m.y);
        const float2 sum = cadd(c, cm), dif = cmi(csub(c, cm));
        a[h] = make_float2(0.5f * sum.x, 0.5f * sum.y);
        b[h] = make_float2(0.5f * dif.x, 0.5f * dif.y);
      }
    }
    __stcs(reinterpret_cast<float4*>(out + (pen0 + 2 * q) * P + k0), make_float4(a[0].x, a[0].y, a[1].x, a[1].y));
    if (2 * q + 1 < npen)
      __stcs(reinterpret_cast<float4*>(out + (pen0 + 2 * q + 1) * P + k0),
             make_float4(b[0].x, b[0].y, b[1].x, b[1].y));
  }
}

// z pass of the packed transform: PAIRS complex columns per CTA, column (x', y)
// of the packed field (G = 2: pencil (x', y) of both meshes; G = 1: pencils
// (2x', y) and (2x'+1, y)).  The CTA takes PACK_W planes x PAIRS / PACK_W rows,
// so it fills whole lines of the interleaved planes.  The last stage stores
// Z[kz] to slab 0 and / or the mirrored entry of slab 1 straight from registers.
template <int N, int G, int PAIRS>
__global__ void __launch_bounds__(PAIRS * N / 16)
fftz_packed_kernel(const float* __restrict__ mesh, float2* __restrict__ out, int kz_cols,
                   const float2* __restrict__ tw) {
  pdl_wait();
  constexpr int NT = PAIRS * N / 16;
  constexpr int CP = PAIRS / 2;
  constexpr int NX = G == 2 ? N : N / 2;
  constexpr int P = zpitch(N);
  constexpr long long IM = G == 2 ? (long long)N * N * N : (long long)N * N;   // from the real to the imaginary pencil
  static_assert(PAIRS % PACK_W == 0 && N % (PAIRS / PACK_W) == 0, "whole blocks of rows");
  extern __shared__ __align__(16) float4 s4[];    // [CP][N] slots of two columns
  const int tid = threadIdx.x;
  using R = fft::PackedRows<N>;
  constexpr int ROWS = PAIRS / PACK_W;
  const int x = blockIdx.x / (N / ROWS) * PACK_W, y = blockIdx.x % (N / ROWS) * ROWS;
  constexpr long long XM = G == 2 ? (long long)N * N : 2LL * N * N;   // mesh: from one packed plane to the next
  const float* base = mesh + x * XM + (long long)y * N;
  float2* o0 = out + R::at(x, y);
  float2* o1 = o0 + (long long)NX * N * P;
  auto gin = [base](int j, int cp) {
    const float* b = base + 2 * cp % PACK_W * XM + 2 * cp / PACK_W * N + j;    // planes 2cp % PACK_W and the next
    constexpr float S = fft::PACK_SCALE<G>;
    return make_float4(S * __ldcg(b), S * __ldcg(b + IM), S * __ldcg(b + XM), S * __ldcg(b + IM + XM));
  };
  auto sin_ = [](int j, int cp) { return s4[cp * N + zsw(j)]; };
  auto sout = [](int j, int cp, float4 v) { s4[cp * N + zsw(j)] = v; };
  auto gout = [o0, o1, kz_cols](int k, int cp, float4 v) {
    const int c = 2 * cp / PACK_W * R::ROW + 2 * cp % PACK_W * 8;
    fft::store_packed<N>(o0 + c, o1 + c, 8, kz_cols, k, v);
  };
  fft::run_stages2<N, CP, NT, true, false, false>(gin, sin_, sout, gout, tw, tid);
}

// Interleaved planes a CTA of the packed y passes takes together (below: measured)
template <int N>
constexpr int Y_PLANES = N <= 512 ? 2 : 1;

// ---- y and x passes --------------------------------------------------------
// 8 adjacent kz columns x N rows per CTA, rows `row_stride` complex apart;
// CTA b covers plane (b / nkb) and kz block (b % nkb).  N/2 threads: one
// pair of radix-8 butterflies (two columns) each per stage; the first stage
// loads from HBM and the last stores to HBM (fft_pass.cuh), in place.  Loads
// and stores use the ordinary L2 policy (.cg), so the CTA that takes the other
// half of a line finds it there, which evict-first (.cs) did not, and the
// planes go last to first, as the previous pass wrote the last ones last.
// Rows with interleaved planes (W > 1): a CTA takes SL planes of one block.
// Two grids at 512^3: 0.402 -> 0.327 (policy) -> 0.310 ms (two planes; one by
// one 0.338), 6.2 TB/s; one grid 0.201 -> 0.158; 256^3 0.053 -> 0.041, with as
// many CTAs as fill the SM.  At 1024^3 two planes fill the SM with one CTA
// (3.66 ms) and one by one takes 3.33 ms; rows of one plane took 3.07, which
// the x pass pays for (xbin.cu).  Bound by HBM.
// PRUNE = 1: rows whose wavenumber k has k^2 + (the block's first kz)^2 >
// k2_max are not stored (with k edges up to k_Nyquist, a fifth of them).
// PRUNE = 2: the same with the plane's number in place of kz (real-space rows,
// xi.cu).
template <int N, int PRUNE, int W, int SL = W == 1 ? 1 : Y_PLANES<N>>
__global__ void __launch_bounds__(N / 2 * SL, N >= 256 ? 2048 / (N * SL) : 4)
fft_cols_kernel(float2* __restrict__ data, long long plane_stride, long long row_stride, int nplanes, int nkb,
                int k2_max, const float2* __restrict__ tw) {
  pdl_wait();
  extern __shared__ __align__(16) float2 s[];
  constexpr int WS = W / SL;
  const int grp = blockIdx.x / (WS * nkb), sub = blockIdx.x - grp * WS * nkb;
  const int plane = nplanes - (grp * WS + sub % WS + 1) * SL, kb = sub / WS;
  if (plane < 0) return;
  float2* base = data + (W > 1 ? fft::PackedRows<N, W>::plane(plane) : plane * plane_stride) + kb * 8 * W;
  auto gin = [base, row_stride](int j, int cp) {
    return __ldcg(reinterpret_cast<const float4*>(base + j * row_stride) + cp);
  };
  const int lim = PRUNE == 1 ? k2_max - 64 * kb * kb : k2_max - plane * plane;
  auto gout = [base, row_stride, lim](int j, int cp, float4 v) {
    if (PRUNE) {
      const int k = signed_k(j, N);
      if (k * k > lim) return;
    }
    __stcg(reinterpret_cast<float4*>(base + j * row_stride) + cp, v);
  };
  fft::col_fft<N, SL, N / 2 * SL, false>(s, gin, gout, tw, threadIdx.x);
}

// Inverse of the packed transform along y, in place: rows whose ky^2 + (the
// block's first kz)^2 > k2_max hold nothing and are taken as zeros; every row
// of every x plane is stored.  (An inverse transform is a forward one with
// real and imaginary parts swapped before and after.)
template <int N, int SL = Y_PLANES<N>>
__global__ void __launch_bounds__(N / 2 * SL, N >= 256 ? 2048 / (N * SL) : 4)
fft_cols_inv_kernel(float2* __restrict__ data, int nplanes, int nkb, int k2_max, const float2* __restrict__ tw) {
  pdl_wait();
  extern __shared__ __align__(16) float2 s[];
  using R = fft::PackedRows<N>;
  constexpr int WS = PACK_W / SL;
  const int grp = blockIdx.x / (WS * nkb), sub = blockIdx.x - grp * WS * nkb;
  const int plane = nplanes - (grp * WS + sub % WS + 1) * SL, kb = sub / WS;
  if (plane < 0) return;
  float2* base = data + R::plane(plane) + kb * R::BLOCK;
  const int lim = k2_max - 64 * kb * kb;
  auto gin = [base, lim](int j, int cp) {
    const int k = signed_k(j, N);
    if (k * k > lim) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v = __ldcg(reinterpret_cast<const float4*>(base + (long long)j * R::ROW) + cp);
    return make_float4(v.y, v.x, v.w, v.z);
  };
  auto gout = [base](int j, int cp, float4 v) {
    __stcg(reinterpret_cast<float4*>(base + (long long)j * R::ROW) + cp, make_float4(v.y, v.x, v.w, v.z));
  };
  fft::col_fft<N, SL, N / 2 * SL, false>(s, gin, gout, tw, threadIdx.x);
}

// Inverse z pass of the packed transform: real fields out (the layout of
// fftz_packed_kernel's input), kz >= kz_cols taken as zero.
template <int N, int G, int PAIRS>
__global__ void __launch_bounds__(PAIRS * N / 16)
fftz_unpack_kernel(const float2* __restrict__ spec, float* __restrict__ mesh, int kz_cols,
                   const float2* __restrict__ tw) {
  pdl_wait();
  constexpr int NT = PAIRS * N / 16;
  constexpr int CP = PAIRS / 2;
  constexpr int NX = G == 2 ? N : N / 2;
  constexpr int P = zpitch(N);
  constexpr long long IM = G == 2 ? (long long)N * N * N : (long long)N * N;
  extern __shared__ __align__(16) float4 s4[];    // [CP][N] slots of two columns
  const int tid = threadIdx.x;
  using R = fft::PackedRows<N>;
  constexpr int ROWS = PAIRS / PACK_W;
  const int x = blockIdx.x / (N / ROWS) * PACK_W, y = blockIdx.x % (N / ROWS) * ROWS;
  constexpr long long XM = G == 2 ? (long long)N * N : 2LL * N * N;
  float* base = mesh + x * XM + (long long)y * N;
  const float2* i0 = spec + R::at(x, y);
  const float2* i1 = i0 + (long long)NX * N * P;
  auto gin = [i0, i1, kz_cols](int j, int cp) {
    const int k = j <= N / 2 ? j : N - j;
    if (k >= kz_cols) return make_float4(0.f, 0.f, 0.f, 0.f);
    const float2* b = (j <= N / 2 ? i0 : i1) + 2 * cp / PACK_W * R::ROW + 2 * cp % PACK_W * 8 + R::kz(k);
    const float2 u = __ldcg(b), v = __ldcg(b + 8);
    return make_float4(u.y, u.x, v.y, v.x);
  };
  auto sin_ = [](int j, int cp) { return s4[cp * N + zsw(j)]; };
  auto sout = [](int j, int cp, float4 v) { s4[cp * N + zsw(j)] = v; };
  auto gout = [base](int j, int cp, float4 v) {
    float* b = base + 2 * cp % PACK_W * XM + 2 * cp / PACK_W * N + j;
    __stcs(b, v.y);
    __stcs(b + IM, v.x);
    __stcs(b + XM, v.w);
    __stcs(b + IM + XM, v.z);
  };
  fft::run_stages2<N, CP, NT, true, false, false>(gin, sin_, sout, gout, tw, tid);
}

template <int N>
constexpr int z_pairs() { return N >= 256 ? 8 : 32768 / (N * 8); }   // >= 256 threads
template <int N, int PRUNE, int W>
int launch_cols(float2* data, long long plane_stride, long long row_stride, int nplanes, int nkb, int k2_max,
                const float2* tw, cudaStream_t st) {
  constexpr int SL = W == 1 ? 1 : Y_PLANES<N>;
  const size_t smem = (size_t)SL * fft::ColBlock<N, SL>::SLAB * sizeof(float2);
  auto kc = fft_cols_kernel<N, PRUNE, W, SL>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(kc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GBP_CUDA_TRY(launch_pdl(kc, dim3((unsigned)(nplanes / SL * nkb)), dim3(N / 2 * SL), smem, st, data, plane_stride,
                          row_stride, nplanes, nkb, k2_max, tw));
  return GBP_OK;
}

template <int N>
int run_fft(const float* mesh, float2* spec, int G, const float2* tw, cudaStream_t st) {
  constexpr int PAIRS = z_pairs<N>();
  constexpr int P = zpitch(N);
  constexpr int C = 8;                    // kz columns per CTA in the y and x passes
  const long long npen = (long long)G * N * N;
  {
    const size_t smem = (size_t)PAIRS * N * sizeof(float2);
    auto k = fftz_kernel<N, PAIRS>;
    GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long blocks = (npen + 2 * PAIRS - 1) / (2 * PAIRS);
    GBP_TRACE("fft_z", st);
    GBP_CUDA_TRY(launch_pdl(k, dim3((unsigned)blocks), dim3(PAIRS * N / 16), smem, st, mesh, spec, npen, tw));
  }
  {  // y pass: a plane is one x slab of one grid; rows (y) are P apart
    GBP_TRACE("fft_y", st);
    const int r = launch_cols<N, 0, 1>(spec, (long long)N * P, (long long)P, G * N, P / C, 0, tw, st);
    if (r) return r;
  }
  // x pass: a plane is one y row of one grid; rows (x) are N*P apart
  for (int g = 0; g < G; ++g) {
    GBP_TRACE("fft_x", st);
    const int r =
        launch_cols<N, 0, 1>(spec + (long long)g * N * N * P, (long long)P, (long long)N * P, N, P / C, 0, tw, st);
    if (r) return r;
  }
  return GBP_OK;
}

template <int N, int G>
int run_z_packed(const float* mesh, float2* spec, int kz_cols, const float2* tw, cudaStream_t st) {
  constexpr int PAIRS = z_pairs<N>();
  constexpr int NX = G == 2 ? N : N / 2;
  const size_t smem = (size_t)PAIRS * N * sizeof(float2);
  auto k = fftz_packed_kernel<N, G, PAIRS>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GBP_TRACE("fft_z", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3((unsigned)(NX * N / PAIRS)), dim3(PAIRS * N / 16), smem, st, mesh, spec, kz_cols,
                          tw));
  return GBP_OK;
}

template <int N>
int run_y_packed(int G, bool rows, float2* spec, int kz_cols, int k2_max, const float2* tw, cudaStream_t st) {
  constexpr int P = zpitch(N);
  if (kz_cols == 0) return GBP_OK;
  GBP_TRACE("fft_y", st);
  // a plane is one x' of one slab: two slabs of N (two grids) or N/2 planes
  if (rows) return launch_cols<N, 1, 1>(spec, (long long)N * P, (long long)P, G * N, kz_cols / 8, k2_max, tw, st);
  using R = fft::PackedRows<N>;
  return launch_cols<N, 1, PACK_W>(spec, 0, (long long)R::ROW, G * N, kz_cols / 8, k2_max, tw, st);
}

template <int N>
int run_y_shells(float2* spec, int nplanes, int r2_max, const float2* tw, cudaStream_t st) {
  constexpr int P = zpitch(N);
  if (nplanes == 0) return GBP_OK;
  GBP_TRACE("fft_y", st);
  return launch_cols<N, 2, 1>(spec, (long long)N * P, (long long)P, nplanes, P / 8, r2_max, tw, st);
}

template <int N>
int run_y_inverse(int G, float2* spec, int kz_cols, int k2_max, const float2* tw, cudaStream_t st) {
  if (kz_cols == 0) return GBP_OK;
  constexpr int SL = Y_PLANES<N>;
  const size_t smem = (size_t)SL * fft::ColBlock<N, SL>::SLAB * sizeof(float2);
  auto k = fft_cols_inv_kernel<N, SL>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GBP_TRACE("fft_y_inverse", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3((unsigned)(G * N / SL * (kz_cols / 8))), dim3(N / 2 * SL), smem, st, spec,
                          G * N, kz_cols / 8, k2_max, tw));
  return GBP_OK;
}

template <int N, int G>
int run_z_unpack(const float2* spec, float* mesh, int kz_cols, const float2* tw, cudaStream_t st) {
  constexpr int PAIRS = z_pairs<N>();
  constexpr int NX = G == 2 ? N : N / 2;
  const size_t smem = (size_t)PAIRS * N * sizeof(float2);
  auto k = fftz_unpack_kernel<N, G, PAIRS>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GBP_TRACE("fft_z_inverse", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3((unsigned)(NX * N / PAIRS)), dim3(PAIRS * N / 16), smem, st, spec, mesh, kz_cols,
                          tw));
  return GBP_OK;
}

}  // namespace

// Entry used by gbp_fft_r2c for power-of-two meshes (declared in api.cu).
bool own_fft_supported(int N) { return N == 64 || N == 128 || N == 256 || N == 512 || N == 1024; }
int own_fft_pitch(int N) { return zpitch(N); }

// Twiddles of an N-point transform: exp(-2 pi i e / N) for e < N, then one
// table per stage of span p > 1 (radix R): entry k * 8 + r holds
// exp(-2 pi i r k / (R p)) for r < R (fft_pass.cuh reads them as float4s).
template <int N>
std::vector<float2> twiddle_tables() {
  std::vector<float2> h((size_t)fft::tw_size<N>(), make_float2(0.f, 0.f));
  for (int e = 0; e < N; ++e) {
    const double a = -2.0 * M_PI * (double)e / (double)N;
    h[e] = make_float2((float)cos(a), (float)sin(a));
  }
  using RD = fft::Radices<N>;
  int p = 1;
  for (int st = 0; st < RD::stages; ++st) {
    const int R = st < RD::n8 ? 8 : (RD::tail == 1 ? 2 : 4);
    if (p > 1) {
      for (int k = 0; k < p; ++k)
        for (int r = 0; r < R; ++r) {
          const double a = -2.0 * M_PI * (double)r * (double)k / ((double)R * (double)p);
          h[(size_t)fft::tw_off<N>(p) + (size_t)k * 8 + r] = make_float2((float)cos(a), (float)sin(a));
        }
    }
    p *= R;
  }
  return h;
}

int own_fft_twiddles(int N, float2** d_tw) {
  std::vector<float2> h;
  switch (N) {
    case 32: h = twiddle_tables<32>(); break;
    case 64: h = twiddle_tables<64>(); break;
    case 128: h = twiddle_tables<128>(); break;
    case 256: h = twiddle_tables<256>(); break;
    case 512: h = twiddle_tables<512>(); break;
    case 1024: h = twiddle_tables<1024>(); break;
    default: return GBP_ERR_UNSUPPORTED;
  }
  float2* d = nullptr;
  if (cudaMalloc(&d, h.size() * sizeof(float2)) != cudaSuccess) return GBP_ERR_ALLOC;
  const cudaError_t ce = cudaMemcpy(d, h.data(), h.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (ce != cudaSuccess) {
    set_last_cuda_error(ce);
    cudaFree(d);
    return GBP_ERR_CUDA;
  }
  *d_tw = d;
  return GBP_OK;
}

int own_fft_r2c(int N, int G, const float* mesh, float2* spec, const float2* tw, cudaStream_t st) {
  switch (N) {
    case 64: return run_fft<64>(mesh, spec, G, tw, st);
    case 128: return run_fft<128>(mesh, spec, G, tw, st);
    case 256: return run_fft<256>(mesh, spec, G, tw, st);
    case 512: return run_fft<512>(mesh, spec, G, tw, st);
    case 1024: return run_fft<1024>(mesh, spec, G, tw, st);
    default: return GBP_ERR_UNSUPPORTED;
  }
}

int own_fft_z_packed(int N, int G, const float* mesh, float2* spec, int kz_cols, const float2* tw,
                     cudaStream_t st) {
#define GBP_Z(NN) \
  case NN:       \
    return G == 2 ? run_z_packed<NN, 2>(mesh, spec, kz_cols, tw, st) : run_z_packed<NN, 1>(mesh, spec, kz_cols, tw, st)
  switch (N) {
    GBP_Z(64);
    GBP_Z(128);
    GBP_Z(256);
    GBP_Z(512);
    GBP_Z(1024);
    default: return GBP_ERR_UNSUPPORTED;
  }
#undef GBP_Z
}

int own_fft_y_packed(int N, int G, float2* spec, int kz_cols, int k2_max, const float2* tw, cudaStream_t st) {
  switch (N) {
    case 64: return run_y_packed<64>(G, false, spec, kz_cols, k2_max, tw, st);
    case 128: return run_y_packed<128>(G, false, spec, kz_cols, k2_max, tw, st);
    case 256: return run_y_packed<256>(G, false, spec, kz_cols, k2_max, tw, st);
    case 512: return run_y_packed<512>(G, false, spec, kz_cols, k2_max, tw, st);
    case 1024: return run_y_packed<1024>(G, false, spec, kz_cols, k2_max, tw, st);
    default: return GBP_ERR_UNSUPPORTED;
  }
}

int own_fft_y_rows(int N, int nplanes, float2* spec, int kz_cols, int k2_max, const float2* tw, cudaStream_t st) {
  switch (N) {
    case 64: return run_y_packed<64>(nplanes / N, true, spec, kz_cols, k2_max, tw, st);
    case 128: return run_y_packed<128>(nplanes / N, true, spec, kz_cols, k2_max, tw, st);
    case 256: return run_y_packed<256>(nplanes / N, true, spec, kz_cols, k2_max, tw, st);
    case 512: return run_y_packed<512>(nplanes / N, true, spec, kz_cols, k2_max, tw, st);
    case 1024: return run_y_packed<1024>(nplanes / N, true, spec, kz_cols, k2_max, tw, st);
    default: return GBP_ERR_UNSUPPORTED;
  }
}

int own_fft_y_inverse(int N, int G, float2* spec, int kz_cols, int k2_max, const float2* tw, cudaStream_t st) {
  switch (N) {
    case 64: return run_y_inverse<64>(G, spec, kz_cols, k2_max, tw, st);
    case 128: return run_y_inverse<128>(G, spec, kz_cols, k2_max, tw, st);
    case 256: return run_y_inverse<256>(G, spec, kz_cols, k2_max, tw, st);
    case 512: return run_y_inverse<512>(G, spec, kz_cols, k2_max, tw, st);
    case 1024: return run_y_inverse<1024>(G, spec, kz_cols, k2_max, tw, st);
    default: return GBP_ERR_UNSUPPORTED;
  }
}

int own_fft_z_unpack(int N, int G, const float2* spec, float* mesh, int kz_cols, const float2* tw, cudaStream_t st) {
#define GBP_Z(NN) \
  case NN:       \
    return G == 2 ? run_z_unpack<NN, 2>(spec, mesh, kz_cols, tw, st) : run_z_unpack<NN, 1>(spec, mesh, kz_cols, tw, st)
  switch (N) {
    GBP_Z(64);
    GBP_Z(128);
    GBP_Z(256);
    GBP_Z(512);
    GBP_Z(1024);
    default: return GBP_ERR_UNSUPPORTED;
  }
#undef GBP_Z
}

int own_fft_y_shells(int N, float2* spec, int nplanes, int r2_max, const float2* tw, cudaStream_t st) {
  switch (N) {
    case 64: return run_y_shells<64>(spec, nplanes, r2_max, tw, st);
    case 128: return run_y_shells<128>(spec, nplanes, r2_max, tw, st);
    case 256: return run_y_shells<256>(spec, nplanes, r2_max, tw, st);
    case 512: return run_y_shells<512>(spec, nplanes, r2_max, tw, st);
    case 1024: return run_y_shells<1024>(spec, nplanes, r2_max, tw, st);
    default: return GBP_ERR_UNSUPPORTED;
  }
}

}  // namespace gbp
