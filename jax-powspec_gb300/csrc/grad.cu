// Gradients of the P_l(k) estimator with respect to particle positions and
// weights (the adjoint of deposit -> R2C -> |delta_k|^2 L_l binning), the
// derivative the reference obtains from JAX autodiff (tests/lognormal.py:
// 60-103 differentiates a loss of powspec_vec through cic_mas_vec).
//
// With P_l(b) = (2l+1) norm / n_b sum_{k in b} c2(k) L_l(mu_k) |D(k)|^2
// (D = F for one grid, D = (F0 + phi F1) / 2 interlaced, phi = exp(i pi
// (kx+ky+kz) / N), norm = L^3 / M^2, the k = 0 mode excluded) and an
// upstream gradient g = dLoss/dP_l(b):
//
//   dLoss/d rho_0(c) = Re sum_{k in half} 2 f A(k) D(k) exp(+i k.c)
//   dLoss/d rho_1(c) = Re sum_{k in half} 2 f A(k) D(k) conj(phi) exp(+i k.c)
//
// with A(k) = sum_l g_{b(k), l} (2l+1) L_l(mu) c2(k) norm / n_b, f = 1 for
// one grid and 1/2 for each of two.  A C2R of the half spectrum counts every
// kz in (0, N/2) twice and the kz = 0, N/2 planes once, so the adjoint
// spectrum is H = f A D (times conj(phi)) with the two planes doubled, and
// gradient mesh = C2R(H) (unnormalised, as the forward transform).
//
// For the library's transform sizes the same adjoint runs on the packed
// transform (gbp_power_backward_packed): the spectrum the fused forward pass
// leaves after its y pass is transformed along x an item at a time (xpass.cuh),
// turned into the packed adjoint spectrum in shared memory and transformed
// back along x in the same kernel; the inverse y and z passes write the
// gradient meshes.  Columns beyond the last k edge are neither stored nor read.
//
// The deposit's adjoint is a gather: for each particle, the B-spline weights
// W and their derivatives dW/du of its stencil nodes (per grid), times the
// gradient mesh there: dLoss/dw_i = sum grad W, dLoss/du_a = w_i sum grad
// dW/du_a, and dLoss/dx_a = inv_cell dLoss/du_a.  The explicit dependence of
// the normalisation and of the shot noise on the weights is two numbers per
// call (grad_coef_kernel, or gbpowspec/grad.py on the cuFFT path), which the
// gather adds to dLoss/dw_i.
#include <cufft.h>
#include <math.h>

#include <algorithm>

#include "xpass.cuh"

namespace gbp {
namespace {

__device__ __forceinline__ int bin_search(const int* __restrict__ thr, int nbe, int nb, int tu, int k2) {
  if (k2 > tu) return -1;
  int lo = 0, hi = nbe + 1;                      // count thresholds <= k2
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(thr + mid) <= k2) lo = mid + 1;
    else hi = mid;
  }
  const int r = lo;
  return min(min(r, nb), nbe) - 1;
}

// (2l+1) dLoss/dP_l norm / n_b of one bin (0 for an empty one).
__device__ __forceinline__ float4 adjoint_coef(const double* __restrict__ grad_pk,
                                               const long long* __restrict__ nmodes, double m, double box, int b) {
  if (nmodes[b] <= 0) return make_float4(0.f, 0.f, 0.f, 0.f);
  const double norm = box * box * box / (m * m) / (double)nmodes[b];
  return make_float4((float)(grad_pk[b * 3 + 0] * norm), 5.0f * (float)(grad_pk[b * 3 + 1] * norm),
                     9.0f * (float)(grad_pk[b * 3 + 2] * norm), 0.0f);
}

// H_g(k) for every half-spectrum entry (row padding -> 0): a warp per z row,
// the per-bin factors (double precision) once per block in shared memory
// when they fit (n_coef = nb, else 0 and each mode forms its own).  0.278 ->
// 0.05 ms at 256^3 with two grids, against a thread per entry that divided
// its index and formed the factors in double for every mode.
constexpr int GS_THREADS = 256;
__global__ void __launch_bounds__(GS_THREADS)
grad_spec_kernel(const float2* __restrict__ spec, float2* __restrict__ hspec, int N, int P, int G,
                 const int* __restrict__ thr, int nbe, int nb, int tu, const float* __restrict__ inv_sinc2,
                 const float2* __restrict__ eph, int mas_order, const double* __restrict__ grad_pk,
                 const long long* __restrict__ nmodes, const double* __restrict__ mass, double box, int n_coef) {
  extern __shared__ float4 s_coef[];
  const double m = mass[0];
  for (int b = threadIdx.x; b < n_coef; b += GS_THREADS) s_coef[b] = adjoint_coef(grad_pk, nmodes, m, box, b);
  __syncthreads();
  const long long total = (long long)N * N * P;
  const int warps = gridDim.x * (GS_THREADS / 32), lane = threadIdx.x & 31;
  for (int row = blockIdx.x * (GS_THREADS / 32) + (threadIdx.x >> 5); row < N * N; row += warps) {
    const int ix = row / N, iy = row - ix * N;
    const int kx = signed_k(ix, N), ky = signed_k(iy, N);
    const int ax = kx < 0 ? -kx : kx, ay = ky < 0 ? -ky : ky;
    float cxy = 1.0f;
    for (int p = 0; p < mas_order; ++p) cxy *= inv_sinc2[ax] * inv_sinc2[ay];
    float2 exy = make_float2(1.f, 0.f);
    if (G == 2) {
      float2 ex = eph[ax], ey = eph[ay];
      if (kx < 0) ex.y = -ex.y;
      if (ky < 0) ey.y = -ey.y;
      exy = make_float2(ex.x * ey.x - ex.y * ey.y, ex.x * ey.y + ex.y * ey.x);
    }
    for (int kz = lane; kz < P; kz += 32) {
      const long long i = (long long)row * P + kz;
      float2 h0 = make_float2(0.f, 0.f), h1 = make_float2(0.f, 0.f);
      const int k2 = kx * kx + ky * ky + kz * kz;
      const int b = (kz <= N / 2 && k2 > 0) ? bin_search(thr, nbe, nb, tu, k2) : -1;
      if (b >= 0) {
        const float4 q = b < n_coef ? s_coef[b] : adjoint_coef(grad_pk, nmodes, m, box, b);
        const float mu2 = (float)(kz * kz) / (float)k2;
        const float l2 = 1.5f * mu2 - 0.5f, l4 = (35.0f * mu2 * mu2 - 30.0f * mu2 + 3.0f) * 0.125f;
        float c2 = cxy;
        for (int p = 0; p < mas_order; ++p) c2 *= inv_sinc2[kz];
        float2 d = spec[i];
        float2 ph = make_float2(1.f, 0.f);
        float f = (kz == 0 || kz == N / 2) ? 2.0f : 1.0f;
        if (G == 2) {
          const float2 ez = eph[kz];
          ph = make_float2(exy.x * ez.x - exy.y * ez.y, exy.x * ez.y + exy.y * ez.x);
          const float2 f1 = spec[i + total];
          d = make_float2(0.5f * (d.x + (f1.x * ph.x - f1.y * ph.y)), 0.5f * (d.y + (f1.x * ph.y + f1.y * ph.x)));
          f *= 0.5f;
        }
        const float a = (q.x + l2 * q.y + l4 * q.z) * c2 * f;
        h0 = make_float2(a * d.x, a * d.y);
        if (G == 2) h1 = make_float2(h0.x * ph.x + h0.y * ph.y, h0.y * ph.x - h0.x * ph.y);   // * conj(phi)
      }
      hspec[i] = h0;
      if (G == 2) hspec[i + total] = h1;
    }
  }
}

// Per-bin factors of the adjoint, (2l+1) dLoss/dP_l norm / n_b as floats, and
// the two explicit dependences of P_l on the weights: scal[0] = dLoss/dM
// through norm = L^3/M^2, scal[1] = -2 L^3/M^2 dLoss/dP_0 (shot noise, times
// w_i).  One block.  A gradient into an empty bin or NaN counts as 0.
constexpr int COEF_THREADS = 256;
__global__ void __launch_bounds__(COEF_THREADS)
grad_coef_kernel(const double* __restrict__ grad_pk, const double* __restrict__ pk,
                 const long long* __restrict__ nmodes, const double* __restrict__ mass, int nb, double box, int shot,
                 float4* __restrict__ coef, double* __restrict__ scal) {
  pdl_wait();
  __shared__ double s_sum[2][COEF_THREADS];
  const double m = mass[0], box3 = box * box * box;
  double dm = 0.0, dq = 0.0;
  for (int b = threadIdx.x; b < nb; b += COEF_THREADS) {
    const double norm = nmodes[b] > 0 ? box3 / (m * m) / (double)nmodes[b] : 0.0;
    float c[3];
    for (int l = 0; l < 3; ++l) {
      const double p = pk[3 * b + l];
      double g = grad_pk[3 * b + l];
      if (isnan(g) || !isfinite(p)) g = 0.0;
      else if (isinf(g)) g = copysign(1.7976931348623157e308, g);
      dm += g * (-2.0 * (isnan(p) ? 0.0 : (isinf(p) ? copysign(1.7976931348623157e308, p) : p)) / m);
      if (l == 0) dq += g;
      c[l] = (float)(g * norm);
    }
    coef[b] = make_float4(c[0], 5.0f * c[1], 9.0f * c[2], 0.0f);
  }
  s_sum[0][threadIdx.x] = dm;
  s_sum[1][threadIdx.x] = dq;
  __syncthreads();
  for (int o = COEF_THREADS / 2; o > 0; o >>= 1) {                  // fixed order
    if (threadIdx.x < o) {
      s_sum[0][threadIdx.x] += s_sum[0][threadIdx.x + o];
      s_sum[1][threadIdx.x] += s_sum[1][threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    scal[0] = s_sum[0][0];
    scal[1] = shot ? -2.0 * box3 / (m * m) * s_sum[1][0] : 0.0;
  }
}

// Packed adjoint spectrum, one item per step: forward x transform, H in place
// (the four values of a pair of modes +-kx, or of two such pairs with one
// grid, are one thread's), inverse x transform (a forward one with real and
// imaginary parts swapped) into `out`, the layout of the input.
template <int N, bool INTER>
__global__ void __launch_bounds__(XLayout<N, INTER>::NT, N >= 1024 && INTER ? 1 : 1024 / XLayout<N, INTER>::NT)
grad_x_kernel(PowGeom g, const float4* __restrict__ coef, float2* __restrict__ out) {
  pdl_wait();
  using L = XLayout<N, INTER>;
  constexpr int TST = L::TST, NX = L::NX, NT = L::NT, H = N / 2, M2 = L::M2;
  extern __shared__ __align__(16) unsigned char smem[];
  float2* s = reinterpret_cast<float2*>(smem);
  const Smem t = load_tables<1, INTER>(g, smem + L::data_bytes());
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int it = blockIdx.x; it < g.items; it += gridDim.x) {
    const int code = __ldg(g.item_list + it), y = code / XITEM_KB, kb = code % XITEM_KB;
    x_forward<N, INTER, false>(s, g.s0, y, kb, g.twx, tid);
    const int c = warp / L::HALVES, kz = kb * XB_C + c;
    const int ky = signed_k(y, N), ay = ky < 0 ? -ky : ky;
    if (kz <= H) {
      float2* a = s + c * TST;
      float2* b = s + (XB_C + c) * TST;
      const bool plane = kz == 0 || kz == H;       // both k and -k are modes of the half spectrum
      const float cyz = t.c2[ay] * t.c2[kz];
      const int kyz2 = ky * ky + kz * kz;
      const float fz2 = (float)(kz * kz);
      // A(k) = sum_l coef_l L_l c2 of the modes +-kx = +-p
      auto amp = [&](int p) {
        const int k2 = p * p + kyz2;
        const int bin = k2 > 0 ? bin_of(g, t, k2) : -1;
        if (bin < 0) return 0.0f;
        const float4 q = __ldg(coef + bin);
        const float mu2 = fz2 / (float)k2;
        const float l2 = 1.5f * mu2 - 0.5f, l4 = (35.0f * mu2 * mu2 - 30.0f * mu2 + 3.0f) * 0.125f;
        return (q.x + l2 * q.y + l4 * q.z) * (cyz * t.c2[p]);
      };
      auto at = [](int x) { return xswz<M2>(x & (NX - 1)); };
      auto cscale = [](float2 v, float f) { return make_float2(v.x * f, v.y * f); };
      auto conj = [](float2 v) { return make_float2(v.x, -v.y); };
      if constexpr (INTER) {
        // exp(i pi k / N) of ky (signed), of -ky (N/2 is its own mirror) and of kz
        const float2 e = t.eph[ay], ez = t.eph[kz];
        const float2 ey = make_float2(e.x, ky < 0 ? -e.y : e.y);
        const float2 eym = make_float2(e.x, ay == H ? ey.y : -ey.y);
        const float2 eyz = fft::cmul(ey, ez), emz = fft::cmul(eym, ez);
        for (int p = lane + 32 * (warp % L::HALVES); p <= H; p += 32 * L::HALVES) {
          const float A = amp(p) * 0.5f;           // f = 1/2
          const float2 ep = t.eph[p], em = make_float2(ep.x, p == H ? ep.y : -ep.y);
          const float2 zp = a[at(p)], zm = a[at(-p)], wp = b[at(p)], wm = b[at(-p)];
          // H0, H1 = H0 conj(phi) of a mode with Z(k) = u, Z(-k) = v
          auto adjoint = [&](float2 u, float2 v, float2 ph, float2 phm, float2& h0, float2& h1) {
            h0 = cscale(unpack_mode(u, v, ph.x, ph.y), A);
            h1 = fft::cmul(h0, conj(ph));
            if (plane) {
              const float2 m0 = cscale(unpack_mode(v, u, phm.x, phm.y), A);
              h0 = fft::cadd(h0, conj(m0));
              h1 = fft::cadd(h1, conj(fft::cmul(m0, conj(phm))));
            }
          };
          float2 h0, h1, k0, k1;
          adjoint(zp, wm, fft::cmul(ep, eyz), fft::cmul(em, emz), h0, h1);     // kx = p
          adjoint(zm, wp, fft::cmul(em, eyz), fft::cmul(ep, emz), k0, k1);     // kx = -p
          a[at(p)] = make_float2(h0.x - h1.y, h0.y + h1.x);
          b[at(-p)] = make_float2(h0.x + h1.y, h1.x - h0.y);
          if (p > 0 && p < H) {
            a[at(-p)] = make_float2(k0.x - k1.y, k0.y + k1.x);
            b[at(p)] = make_float2(k0.x + k1.y, k1.x - k0.y);
          }
        }
      } else {
        const float f = plane ? 2.0f : 1.0f;       // the planes twice
        for (int p = lane + 32 * (warp % L::HALVES); p <= N / 4; p += 32 * L::HALVES) {
          const int r = H - p;
          const float Ap = amp(p) * f, Ar = amp(r) * f;
          const float2 wp = __ldg(g.tw + p), wr = __ldg(g.tw + r);
          const float2 ap = a[at(p)], ar = a[at(r)], bp = b[at(p)], br = b[at(r)];
          const float2 ha = cscale(unpack_mode(ap, br, wp.x, wp.y), Ap);       // kx = p
          const float2 hd = cscale(unpack_mode(ar, bp, wp.x, -wp.y), Ap);      // kx = -p
          const float2 hc = cscale(unpack_mode(ar, bp, wr.x, wr.y), Ar);       // kx = r
          const float2 hb = cscale(unpack_mode(ap, br, wr.x, -wr.y), Ar);      // kx = -r = p + N/2
          auto pack = [&](float2 u, float2 v, float2 w) {                      // u + v + i conj(w) (u - v)
            const float2 d = fft::cmul(fft::csub(u, v), conj(w));
            return make_float2(u.x + v.x - d.y, u.y + v.y + d.x);
          };
          a[at(p)] = pack(ha, hb, wp);
          b[at(p)] = pack(conj(hd), conj(hc), wp);
          if (p > 0) {
            a[at(r)] = pack(hc, hd, wr);
            b[at(r)] = pack(conj(hb), conj(ha), wr);
          }
        }
      }
    }
    __syncthreads();
    auto gin = [s](int x, int cp) {
      const float2 u = s[(2 * cp) * TST + xswz<M2>(x)], v = s[(2 * cp + 1) * TST + xswz<M2>(x)];
      return make_float4(u.y, u.x, v.y, v.x);
    };
    using R = fft::PackedRows<N>;
    float2* dst = out + kb * R::BLOCK;
    const long long r0 = (long long)y * R::ROW, r1 = R::plane(NX) + (long long)((N - y) & (N - 1)) * R::ROW;
    auto gout = [dst, r0, r1](int x, int cp, float4 v) {
      __stcs(reinterpret_cast<float4*>(dst + (cp < 4 ? r0 : r1) + R::plane(x)) + (cp & 3),
             make_float4(v.y, v.x, v.w, v.z));
    };
    fft::col_fft<NX, 2, NT, false, decltype(gin), decltype(gout), true>(s, gin, gout, g.twx, tid);
    __syncthreads();
  }
}

template <int N, bool INTER>
int launch_grad_x(PowGeom g, const float4* coef, float2* out, cudaStream_t st) {
  using L = XLayout<N, INTER>;
  g.warps = 0;                                     // no bins in shared memory
  const size_t smem = L::data_bytes() + smem_plan(N, g.nbe, g.lut_n, 0, 1).total;
  if (smem > 227 * 1024) return GBP_ERR_UNSUPPORTED;
  auto k = grad_x_kernel<N, INTER>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GBP_TRACE("grad_x", st);
  GBP_CUDA_TRY(launch_pdl(k, dim3(std::max(1, std::min(g.items, 1216))), dim3(L::NT), smem, st, g, coef, out));
  return GBP_OK;
}

// B-spline of order MAS at grid coordinate u (+ half a cell for the second
// grid): first node, weights and their derivatives d/du.  Same node
// convention and arithmetic as the deposit kernels.
template <int MAS>
__device__ __forceinline__ void bspline_dw(float u, int N, int half, int& first, float (&w)[MAS], float (&dw)[MAS]) {
  const float fu = floorf(u);
  float d = __fsub_rn(u, fu);
  int i = pmod(__float2int_rz(fu), N);
  if (half) {
    d = __fadd_rn(d, 0.5f);
    if (d >= 1.0f) { d = __fsub_rn(d, 1.0f); i += 1; }
  }
  if constexpr (MAS == GBP_NGP) {
    first = i + (d >= 0.5f ? 1 : 0);
    w[0] = 1.0f;
    dw[0] = 0.0f;
  } else if constexpr (MAS == GBP_CIC) {
    first = i;
    w[0] = 1.0f - d; w[1] = d;
    dw[0] = -1.0f; dw[1] = 1.0f;
  } else if constexpr (MAS == GBP_TSC) {
    const int up = d >= 0.5f ? 1 : 0;
    const float s = up ? d - 1.0f : d;
    first = i + up - 1;
    const float l = 0.5f - s, r = 0.5f + s;
    w[0] = 0.5f * l * l; w[1] = 0.75f - s * s; w[2] = 0.5f * r * r;
    dw[0] = -l; dw[1] = -2.0f * s; dw[2] = r;
  } else {
    const float t = d, m = 1.0f - d;
    const float c6 = 1.0f / 6.0f;
    first = i - 1;
    w[0] = m * m * m * c6;
    w[1] = (4.0f - 6.0f * t * t + 3.0f * t * t * t) * c6;
    w[2] = (4.0f - 6.0f * m * m + 3.0f * m * m * m) * c6;
    w[3] = t * t * t * c6;
    dw[0] = -0.5f * m * m;
    dw[1] = (-12.0f * t + 9.0f * t * t) * c6;
    dw[2] = (12.0f * m - 9.0f * m * m) * c6;
    dw[3] = 0.5f * t * t;
  }
}

// A z row of the stencil is read where it lies when it does not wrap.
// scal (nullable): adds the explicit weight dependences (grad_coef_kernel) to
// grad_w in double, rounded once.
template <int MAS, int G>
__global__ void __launch_bounds__(256)
deposit_gather_kernel(const float* __restrict__ x, const float* __restrict__ y, const float* __restrict__ z,
                      const float* __restrict__ wts, long long n, float ox, float oy, float oz, float inv_cell, int N,
                      const float* __restrict__ grad_mesh, const double* __restrict__ scal, float* gx, float* gy,
                      float* gz, float* gw) {
  pdl_wait();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float u[3] = {__fmul_rn(__fsub_rn(x[i], ox), inv_cell), __fmul_rn(__fsub_rn(y[i], oy), inv_cell),
                      __fmul_rn(__fsub_rn(z[i], oz), inv_cell)};
  const float wi = wts ? wts[i] : 1.0f;
  const long long M = (long long)N * N * N;
  float sw = 0.f, su[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int g = 0; g < G; ++g) {
    int f[3];
    float w[3][MAS], dw[3][MAS];
#pragma unroll
    for (int a = 0; a < 3; ++a) bspline_dw<MAS>(u[a], N, g, f[a], w[a], dw[a]);
    const float* gm = grad_mesh + g * M;
    int cz[MAS];
#pragma unroll
    for (int r = 0; r < MAS; ++r) cz[r] = wrap_index(f[2] + r, N);
#pragma unroll
    for (int rx = 0; rx < MAS; ++rx) {
      const long long cx = (long long)wrap_index(f[0] + rx, N) * N;
#pragma unroll
      for (int ry = 0; ry < MAS; ++ry) {
        const float* row = gm + (cx + wrap_index(f[1] + ry, N)) * N;
        float v = 0.f, d = 0.f;                      // the row's value and z derivative
#pragma unroll
        for (int rz = 0; rz < MAS; ++rz) {
          const float gv = __ldg(row + cz[rz]);
          v += gv * w[2][rz];
          d += gv * dw[2][rz];
        }
        const float wxy = w[0][rx] * w[1][ry];
        sw += wxy * v;
        su[0] += dw[0][rx] * w[1][ry] * v;
        su[1] += w[0][rx] * dw[1][ry] * v;
        su[2] += wxy * d;
      }
    }
  }
  gx[i] = wi * su[0] * inv_cell;
  gy[i] = wi * su[1] * inv_cell;
  gz[i] = wi * su[2] * inv_cell;
  if (gw) gw[i] = scal ? (float)((double)sw + scal[0] + (double)wi * scal[1]) : sw;
}

template <int MAS>
int launch_gather(const float* x, const float* y, const float* z, const float* w, int64_t n, float ox, float oy,
                  float oz, float inv_cell, int N, int G, const float* grad_mesh, const double* scal, float* gx,
                  float* gy, float* gz, float* gw, cudaStream_t st) {
  const dim3 blocks((unsigned)((n + 255) / 256));
  GBP_TRACE("grad_gather", st);
  auto k = G == 2 ? deposit_gather_kernel<MAS, 2> : deposit_gather_kernel<MAS, 1>;
  GBP_CUDA_TRY(launch_pdl(k, blocks, dim3(256), 0, st, x, y, z, w, static_cast<long long>(n), ox, oy, oz, inv_cell, N,
                          grad_mesh, scal, gx, gy, gz, gw));
  return GBP_OK;
}

int gather(const float* x, const float* y, const float* z, const float* w, int64_t n, float xmin, float ymin,
           float zmin, float inv_cell, int N, int mas, int interlace, const float* grad_mesh, const double* scal,
           float* grad_x, float* grad_y, float* grad_z, float* grad_w, cudaStream_t st) {
  if (n < 0 || N < 1 || mas < GBP_NGP || mas > GBP_PCS || !grad_mesh || !grad_x || !grad_y || !grad_z)
    return GBP_ERR_INVALID;
  if (n == 0) return GBP_OK;
  if (!x || !y || !z) return GBP_ERR_INVALID;
  const int G = interlace ? 2 : 1;
#define GBP_GATHER(M) \
  launch_gather<M>(x, y, z, w, n, xmin, ymin, zmin, inv_cell, N, G, grad_mesh, scal, grad_x, grad_y, grad_z, grad_w, st)
  switch (mas) {
    case GBP_NGP: return GBP_GATHER(GBP_NGP);
    case GBP_CIC: return GBP_GATHER(GBP_CIC);
    case GBP_TSC: return GBP_GATHER(GBP_TSC);
    default: return GBP_GATHER(GBP_PCS);
  }
#undef GBP_GATHER
}

}  // namespace
}  // namespace gbp

using namespace gbp;

extern "C" int gbp_power_backward_workspace_size(gbp_fft_plan plan, size_t* bytes) {
  if (!plan || !bytes) return GBP_ERR_INVALID;
  cufftHandle h;
  size_t w = 0;
  const int st = c2r_plan(plan->n, plan->pitch, 1, &h, &w);
  if (st) return st;
  *bytes = align256((size_t)plan->grids * plan->n * plan->n * plan->pitch * sizeof(float2)) + align256(w > 0 ? w : 1);
  return GBP_OK;
}

extern "C" int gbp_power_backward(const void* spectrum, gbp_fft_plan plan, gbp_bins B, int mas_order,
                                  const double* grad_pk, const long long* nmodes, const double* mass, double box_size,
                                  float* grad_mesh, void* workspace, size_t ws_bytes, gbp_stream_t stream_) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  if (!spectrum || !plan || !B || !grad_pk || !nmodes || !mass || !grad_mesh || !(box_size > 0.0))
    return GBP_ERR_INVALID;
  if (plan->n != B->N || plan->grids < 1 || plan->grids > 2 || mas_order < 0 || mas_order > 8) return GBP_ERR_INVALID;
  const int N = plan->n, P = plan->pitch, G = plan->grids;
  cufftHandle h;
  size_t w = 0;
  int r = c2r_plan(N, P, 1, &h, &w);
  if (r) return r;
  const long long total = (long long)N * N * P;
  const size_t need = align256((size_t)G * total * sizeof(float2)) + align256(w > 0 ? w : 1);
  if (!workspace || ws_bytes < need) return GBP_ERR_WORKSPACE;
  // The adjoint spectrum first, then a work area of its own (256 bytes when
  // the plan needs none): cuFFT fails to execute with a work area that
  // starts at its input.
  Carver cv(workspace);
  float2* hspec = cv.take<float2>((size_t)G * total);
  void* cws = cv.take<char>(w > 0 ? w : 1);
  {
    GBP_TRACE("grad_spectrum", st);
    const int n_coef = (size_t)B->nb * sizeof(float4) <= 48 * 1024 ? B->nb : 0;
    const int blocks = std::min(1216, (N * N + GS_THREADS / 32 - 1) / (GS_THREADS / 32));
    grad_spec_kernel<<<blocks, GS_THREADS, (size_t)n_coef * sizeof(float4), st>>>(
        static_cast<const float2*>(spectrum), hspec, N, P, G, B->d_thr, B->nbe, B->nb, B->last_closed,
        B->d_inv_sinc2, B->d_eph, mas_order, grad_pk, nmodes, mass, box_size, n_coef);
    GBP_LAUNCH_CHECK();
  }
  GBP_TRACE("grad_c2r", st);
  for (int g = 0; g < G; ++g) {
    r = c2r_exec(N, P, 1, hspec + g * total, grad_mesh + (long long)g * N * N * N, cws, st);
    if (r) return r;
  }
  return GBP_OK;
}

extern "C" int gbp_deposit_backward(const float* x, const float* y, const float* z, const float* w, int64_t n,
                                    float xmin, float ymin, float zmin, float inv_cell, int N, int mas, int interlace,
                                    const float* grad_mesh, float* grad_x, float* grad_y, float* grad_z,
                                    float* grad_w, gbp_stream_t stream_) {
  return gather(x, y, z, w, n, xmin, ymin, zmin, inv_cell, N, mas, interlace, grad_mesh, nullptr, grad_x, grad_y,
                grad_z, grad_w, reinterpret_cast<cudaStream_t>(stream_));
}

extern "C" int gbp_deposit_backward_total(const float* x, const float* y, const float* z, const float* w, int64_t n,
                                          float xmin, float ymin, float zmin, float inv_cell, int N, int mas,
                                          int interlace, const float* grad_mesh, const double* scal, float* grad_x,
                                          float* grad_y, float* grad_z, float* grad_w, gbp_stream_t stream_) {
  if (grad_w && !scal) return GBP_ERR_INVALID;
  return gather(x, y, z, w, n, xmin, ymin, zmin, inv_cell, N, mas, interlace, grad_mesh, scal, grad_x, grad_y, grad_z,
                grad_w, reinterpret_cast<cudaStream_t>(stream_));
}

namespace gbp {
namespace {
size_t packed_bytes(gbp_fft_plan plan) {
  return align256((size_t)plan->grids * plan->n * plan->n * plan->pitch * sizeof(float2));
}
}  // namespace
}  // namespace gbp

extern "C" int gbp_power_backward_packed_workspace_size(gbp_fft_plan plan, gbp_bins B, size_t* bytes) {
  if (!plan || !B || !bytes || plan->n != B->N) return GBP_ERR_INVALID;
  if (!plan->own || (plan->grids != 1 && plan->grids != 2)) return GBP_ERR_UNSUPPORTED;
  *bytes = packed_bytes(plan) + align256((size_t)B->nb * sizeof(float4));
  return GBP_OK;
}

extern "C" int gbp_power_backward_packed(const void* packed, gbp_fft_plan plan, gbp_bins B, int mas_order,
                                         const double* grad_pk, const double* pk, const long long* nmodes,
                                         const double* mass, double box_size, int subtract_shot, float* grad_mesh,
                                         double* scal, void* workspace, size_t ws_bytes, gbp_stream_t stream_) {
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream_);
  if (!packed || !plan || !B || !grad_pk || !pk || !nmodes || !mass || !grad_mesh || !scal || !(box_size > 0.0))
    return GBP_ERR_INVALID;
  if (mas_order < 0 || mas_order > 8) return GBP_ERR_INVALID;
  if ((reinterpret_cast<uintptr_t>(packed) & 15u) != 0) return GBP_ERR_INVALID;
  size_t need = 0;
  int r = gbp_power_backward_packed_workspace_size(plan, B, &need);
  if (r) return r;
  if (!workspace || ws_bytes < need) return GBP_ERR_WORKSPACE;
  const int N = plan->n, G = plan->grids;
  Carver cv(workspace);
  float2* h = cv.take<float2>(packed_bytes(plan) / sizeof(float2));
  float4* coef = cv.take<float4>(B->nb);
  {
    GBP_TRACE("grad_coef", st);
    GBP_CUDA_TRY(launch_pdl(grad_coef_kernel, dim3(1), dim3(COEF_THREADS), 0, st, grad_pk, pk, nmodes, mass, B->nb,
                            box_size, subtract_shot, coef, scal));
  }
  PowGeom g{};
  g.s0 = static_cast<const float2*>(packed);
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
  g.items = B->n_xitems;
  g.item_list = B->d_xitems;
#define GBP_GX(NN) \
  case NN: r = G == 2 ? launch_grad_x<NN, true>(g, coef, h, st) : launch_grad_x<NN, false>(g, coef, h, st); break
  switch (N) {
    GBP_GX(64);
    GBP_GX(128);
    GBP_GX(256);
    GBP_GX(512);
    GBP_GX(1024);
    default: r = GBP_ERR_UNSUPPORTED;
  }
#undef GBP_GX
  if (r) return r;
  r = own_fft_y_inverse(N, G, h, B->kz_cols, B->last_closed, plan->tw, st);
  if (r) return r;
  return own_fft_z_unpack(N, G, h, grad_mesh, B->kz_cols, plan->tw, st);
}
