// What a deposit leaves besides its cells -- integer counters, exact totals and
// per-block float-float weight sums -- and their fold into gbp_deposit_stats.
// The mesh deposit folds them in a kernel of its own (deposit_core.cuh), the
// fused path in a block of power_reduce_kernel (power_core.cuh).
#pragma once

#include <math.h>

#include "gbp_internal.cuh"

namespace gbp {

struct Catalogue {
  const float *x, *y, *z, *w;
  float ox, oy, oz, inv_cell;
};

struct DepCounters {           // zeroed by one memset per call; integers: any order gives the same totals
  unsigned int maxw_bits;
  unsigned int outgrown;       // some tile has more entries than DepGeom::flag_cap
  unsigned long long kept, bad;
  Catalogue cat;               // what the fill kernel read
};

struct StatsFold {
  const DepCounters* ctr;
  const float4* block_stats;   // [nblocks] (sum w, sum w^2) as float-floats
  int nblocks, compat, G;
  const long long* tile_mass;  // [2][ntiles] totals of the tiles' fixed-point cells per grid, at the common scale
  int ntiles;
  gbp_deposit_stats* out;
};

namespace {

// Fixed-point exponent s: one contribution w * W (|W| <= 1, or <= 8 for the
// reference CIC, whose fractions can leave [0,1) off the box) is an integer
// below 2^30 in magnitude, so it fits one 32-bit atomic on the low word; the
// 64-bit cell sums hold n * 2^30 without overflow for any n < 2^32.
// Float32 and integer operations only (GB300's FP64 rate is tiny).
__device__ __forceinline__ int fixed_scale_exp(unsigned maxw_bits, int compat) {
  const float maxw = __uint_as_float(maxw_bits);
  if (!(maxw > 0.0f) || !(maxw < 3.0e38f)) return 0;
  int ew;
  frexpf(maxw, &ew);                            // maxw < 2^ew
  const int s = 30 - ew - (compat ? 3 : 0);
  return s < -100 ? -100 : (s > 100 ? 100 : s);
}

__device__ __forceinline__ ff warp_ff_sum(ff v) {
  for (int o = 16; o > 0; o >>= 1) {
    ff t{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
    v = ff_add(v, t);
  }
  return v;
}

// The block of NT threads stands for STATS_LANES lanes: lane v adds blocks v,
// v + STATS_LANES, ... in that order, each warp of lanes folds by a fixed xor
// tree, thread 0 adds the warps in order, whatever NT (the same bits).
constexpr int STATS_LANES = 1024;

template <int NT>
__device__ __forceinline__ void fold_stats(const StatsFold& f) {
  constexpr int L = STATS_LANES / NT, SU = 4;
  __shared__ ff s_a[STATS_LANES / 32], s_b[STATS_LANES / 32];
#pragma unroll
  for (int j = 0; j < L; ++j) {
    const int lane = threadIdx.x + j * NT;
    ff a{0.f, 0.f}, b{0.f, 0.f};
    for (int k0 = lane; k0 < f.nblocks; k0 += SU * STATS_LANES) {
      float4 v[SU];            // SU loads in flight before the in-order adds
#pragma unroll
      for (int u = 0; u < SU; ++u) {
        const int k = k0 + u * STATS_LANES;
        v[u] = k < f.nblocks ? f.block_stats[k] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < SU; ++u) {
        if (k0 + u * STATS_LANES >= f.nblocks) break;
        a = ff_add(a, ff{v[u].x, v[u].y});
        b = ff_add(b, ff{v[u].z, v[u].w});
      }
    }
    a = warp_ff_sum(a);
    b = warp_ff_sum(b);
    if ((threadIdx.x & 31) == 0) {
      s_a[lane >> 5] = a;
      s_b[lane >> 5] = b;
    }
  }
  __shared__ long long s_m[2][NT / 32];
  long long m[2] = {0, 0};
#pragma unroll 4
  for (int k = threadIdx.x; k < f.ntiles; k += NT) {
    m[0] += f.tile_mass[k];
    if (f.G == 2) m[1] += f.tile_mass[f.ntiles + k];
  }
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    for (int o = 16; o > 0; o >>= 1) m[g] += __shfl_xor_sync(0xffffffffu, m[g], o);
    if ((threadIdx.x & 31) == 0) s_m[g][threadIdx.x >> 5] = m[g];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    ff ta{0.f, 0.f}, tb{0.f, 0.f};
    for (int k = 0; k < STATS_LANES / 32; ++k) {
      ta = ff_add(ta, s_a[k]);
      tb = ff_add(tb, s_b[k]);
    }
    const DepCounters* c = f.ctr;
    const int s = fixed_scale_exp(c->maxw_bits, f.compat);
    const double inv = ldexp(1.0, -s);
    for (int g = 0; g < 2; ++g) {
      long long t = 0;
      for (int k = 0; k < NT / 32; ++k) t += s_m[g][k];
      f.out->mass[g] = g < f.G ? (double)t * inv : 0.0;
    }
    f.out->sum_w = (double)ta.hi + (double)ta.lo;
    f.out->sum_w2 = (double)tb.hi + (double)tb.lo;
    f.out->n_kept = (long long)c->kept;
    f.out->n_nonfinite = (long long)c->bad;
    f.out->scale_exp = s;
    f.out->flags = c->outgrown ? GBP_STATS_REFILLED : 0;
  }
}

}  // namespace
}  // namespace gbp
