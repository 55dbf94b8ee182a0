// Deposit internals shared by the mesh deposit (deposit.cu) and the deposit
// fused with the z pass of the FFT (depfft.cu): geometry, B-spline and
// reference-compatible stencils, tile bucketing in one pass (buckets of a
// fixed capacity and a table for their surplus; count, scan and scatter for a
// large mesh with few particles), int64 fixed-point helpers, statistics and
// workspace layout.
#pragma once

#include <algorithm>
#include <cmath>

#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include "deposit_stats.cuh"
#include "gbp_internal.cuh"

namespace gbp {
namespace {

constexpr int TILE = 16;              // tile edge (cells); >= widest stencil (5)
constexpr int TILE3 = TILE * TILE * TILE;
constexpr int DEP_THREADS = 256;
constexpr int CNT_THREADS = 256;
constexpr int CNT_ITEMS = 2;          // particles per thread in count/scatter
constexpr float MAX_ABS_U = 1073741824.0f;  // |u| < 2^30 cells, else dropped
constexpr int kCubeTiles[3] = {TILE, TILE, TILE};   // mesh deposit: 16^3-cell tiles
// Per-tile counters sit one 128-byte line apart: the bucketing's global
// atomics on different tiles never contend for one L2 line.
constexpr int CSTRIDE = 32;

struct DepGeom {
  const float* x;
  const float* y;
  const float* z;
  const float* w;
  long long n;
  float ox, oy, oz, inv_cell;
  int N;
  int wrap;         // compat modes only
  int td[3];        // tile edge per axis (x, y, z)
  int ts[3];        // log2(td) when td is a power of two, else -1
  int nt[3];        // tiles per axis
  int vec_ok;       // mesh pointers are 16-byte aligned (float4 tile stores allowed)
  const gbp_job* job;  // non-null: particles, n and box geometry are read from here
  long long cap;       // job mode: the capacity the launches were sized for
  unsigned tcap;       // > 0: buckets of a fixed capacity, tile t's at entry t * tcap (fill path)
  unsigned flag_cap;   // entries of a tile beyond which GBP_STATS_REFILLED is reported
  unsigned ccap[4];    // column tiles: capacity of each class's part of a bucket
  unsigned coff[4];    // and where in the bucket it starts
};

// Job mode: the particle pointers, count and box geometry come from a
// gbp_job in device memory (one broadcast load per thread), so the launch
// parameters do not depend on the mock.  A compile-time choice: with the job's
// and the parameters' fields merged at run time the compiler (nvcc 13.0) kept
// the parameters' x beside the job's y, z and n.
template <bool JOB>
__device__ __forceinline__ DepGeom catalogue_of(const DepGeom& gp) {
  DepGeom g = gp;
  if constexpr (JOB) {
    const gbp_job j = *gp.job;
    g.x = j.x; g.y = j.y; g.z = j.z; g.w = j.w;
    g.n = j.n < 0 ? 0 : (j.n > gp.cap ? gp.cap : j.n);   // the buckets hold `cap` particles at most
    g.ox = j.xmin; g.oy = j.ymin; g.oz = j.zmin; g.inv_cell = j.inv_cell;
  }
  return g;
}

// Node index reduced into [0, N).  Stencil nodes lie within a few cells of
// [0, N); tiny meshes fall back to the general modulo.
__device__ __forceinline__ int wrapn(int n, int N) {
  if (N < 8) return pmod(n, N);
  return n < 0 ? n + N : (n >= N ? n - N : n);
}

__device__ __forceinline__ int tile_of(const DepGeom& g, int ax, int node) {
  return g.ts[ax] >= 0 ? (node >> g.ts[ax]) : node / g.td[ax];
}

template <int MAS, int CM>
struct Scheme {
  static constexpr int R = CM ? 2 : MAS;    // nodes per axis
};

// One axis of one particle: nodes first .. first+R-1 (not yet wrapped), their
// weights, and a mask of nodes that are valid scatter indices (only the
// reference-compat variants ever drop nodes).
template <int R>
struct Axis {
  int first;
  unsigned vmask;
  float w[R];
};

// B-spline of order MAS with nodes at integer grid coordinates (the
// reference's node convention: node i sits at xmin + i*H).  `half` shifts
// the particle by +half a cell (the second, interlaced grid).  NC > 0: the
// mesh side as a power-of-two constant (the cell index wraps with a mask,
// the same value as pmod for every int).  Every operation is an intrinsic: as
// plain expressions the compiler chose per kernel instance which products to
// fuse, and two tile shapes of one build could then differ in the last bits
// of their cells (nvcc 13.0 with registers for five CTAs per SM in the
// deposit/z kernel: 64^3 PCS).
template <int MAS, int NC = 0>
__device__ __forceinline__ void axis_bspline(float u, int N, int half, Axis<MAS>& a) {
  static_assert(NC == 0 || (NC & (NC - 1)) == 0, "NC is a power of two");
  const float fu = floorf(u);
  float d = __fsub_rn(u, fu);                 // exact, in [0, 1)
  const int i0 = __float2int_rz(fu);
  int i = NC ? (i0 & (NC - 1)) : wrap_index(i0, N);
  if (half) {
    d = __fadd_rn(d, 0.5f);
    if (d >= 1.0f) { d = __fsub_rn(d, 1.0f); i += 1; }
  }
  a.vmask = (1u << MAS) - 1u;
  if constexpr (MAS == GBP_NGP) {
    a.first = i + (d >= 0.5f ? 1 : 0);
    a.w[0] = 1.0f;
  } else if constexpr (MAS == GBP_CIC) {
    a.first = i;
    a.w[0] = __fsub_rn(1.0f, d);
    a.w[1] = d;
  } else if constexpr (MAS == GBP_TSC) {
    const int up = d >= 0.5f ? 1 : 0;           // nearest node is i+up
    const float s = up ? __fsub_rn(d, 1.0f) : d;  // offset from it, [-0.5, 0.5)
    a.first = i + up - 1;
    const float l = __fsub_rn(0.5f, s), r = __fadd_rn(0.5f, s);
    a.w[0] = __fmul_rn(__fmul_rn(0.5f, l), l);
    a.w[1] = __fmaf_rn(-s, s, 0.75f);
    a.w[2] = __fmul_rn(__fmul_rn(0.5f, r), r);
  } else {                                      // PCS (cubic B-spline)
    const float t = d, m = __fsub_rn(1.0f, d);
    const float c6 = 1.0f / 6.0f;
    a.first = i - 1;
    auto cube = [c6](float v) { return __fmul_rn(__fmul_rn(__fmul_rn(v, v), v), c6); };
    auto inner = [c6](float v) {                // (4 - 6 v^2 + 3 v^3) / 6
      const float q = __fmaf_rn(__fmul_rn(-6.0f, v), v, 4.0f);
      return __fmul_rn(__fmaf_rn(__fmul_rn(__fmul_rn(3.0f, v), v), v, q), c6);
    };
    a.w[0] = cube(m);
    a.w[1] = inner(t);
    a.w[2] = inner(m);
    a.w[3] = cube(t);
  }
}

// The reference CIC along one axis, bit for bit.
//   CM == GBP_COMPAT_VEC follows src/mas.py:103-140 (cic_mas_vec): truncating
//     int32 cast (:107), fraction (:111), wrap = floor-mod of ix+1 (:121);
//     no-wrap zeroes ixp but tests the zeroed value, so the fraction is kept
//     (:125-126).
//   CM == GBP_COMPAT_SCAN follows src/mas.py:44-67 (cic_mas): mdx is computed
//     before the wrap branch (:56); wrap subtracts n once (:24); no-wrap sets
//     both ixp and the fraction to zero (:34).
// Then the scatter's index rule: -N <= idx < 0 maps to idx+N, anything else
// outside [0, N) drops the update (jax .at[].add default mode).
template <int CM>
__device__ __forceinline__ void axis_compat(float u, int N, int wrap, Axis<2>& a) {
  const int ix = __float2int_rz(u);
  const float d = __fsub_rn(u, __int2float_rn(ix));
  const float m = __fsub_rn(1.0f, d);
  int ixp = ix + 1;
  float dh = d;
  if (CM == GBP_COMPAT_VEC) {
    if (wrap) ixp = wrap_index(ixp, N);         // = pmod(ixp + N, N): |ixp| < 2^30 + 1
    else if (ixp >= N) ixp = 0;
  } else {
    if (wrap) { if (ixp >= N) ixp -= N; }
    else if (ixp >= N) { ixp = 0; dh = 0.0f; }
  }
  const bool lo_ok = ix >= -N && ix < N;
  const bool hi_ok = ixp >= -N && ixp < N;
  const int lo = ix < 0 ? ix + N : ix;
  const int hi = ixp < 0 ? ixp + N : ixp;
  // When both are valid, hi == lo + 1 (mod N) in every branch above.
  a.first = lo_ok ? lo : hi - 1;
  a.vmask = (lo_ok ? 1u : 0u) | (hi_ok ? 2u : 0u);
  a.w[0] = m;
  a.w[1] = dh;
}

template <int MAS, int CM, int NC = 0>
__device__ __forceinline__ void make_axis(const DepGeom& g, float u, int grid, Axis<Scheme<MAS, CM>::R>& a) {
  if constexpr (CM != 0) axis_compat<CM>(u, g.N, g.wrap, a);
  else axis_bspline<MAS, NC>(u, g.N, grid, a);
}

// The particles of one thread in count/scatter: loads issued together.
struct Batch {
  float x[CNT_ITEMS], y[CNT_ITEMS], z[CNT_ITEMS], w[CNT_ITEMS];
  bool in[CNT_ITEMS];
};

__device__ __forceinline__ void load_batch(const DepGeom& g, Batch& b, long long blk) {
  const long long base = blk * CNT_THREADS * CNT_ITEMS + threadIdx.x;
#pragma unroll
  for (int k = 0; k < CNT_ITEMS; ++k) {
    const long long i = base + (long long)k * CNT_THREADS;
    b.in[k] = i < g.n;
    if (b.in[k]) {
      b.x[k] = __ldcs(g.x + i);
      b.y[k] = __ldcs(g.y + i);
      b.z[k] = __ldcs(g.z + i);
      b.w[k] = g.w ? __ldcs(g.w + i) : 1.0f;
    }
  }
}

// Grid coordinate of a particle; false if it must be dropped (non-finite, or
// so far outside the box that int32 cells would overflow).
__device__ __forceinline__ bool grid_coords(const DepGeom& g, float x, float y, float z, float u[3]) {
  u[0] = __fmul_rn(__fsub_rn(x, g.ox), g.inv_cell);
  u[1] = __fmul_rn(__fsub_rn(y, g.oy), g.inv_cell);
  u[2] = __fmul_rn(__fsub_rn(z, g.oz), g.inv_cell);
  return fabsf(u[0]) < MAX_ABS_U && fabsf(u[1]) < MAX_ABS_U && fabsf(u[2]) < MAX_ABS_U;  // false for NaN
}

// Distinct tiles touched along one axis by the valid nodes of all grids
// (at most 3 because a stencil spans at most 5 nodes and tiles are wider).
template <int MAS, int G, int CM>
__device__ __forceinline__ int axis_tiles(const DepGeom& g, int ax, float u, int& t0, int& t1, int& t2) {
  constexpr int R = Scheme<MAS, CM>::R;
  constexpr int W = R + (G - 1);
  Axis<R> a;
  make_axis<MAS, CM>(g, u, 0, a);
  int lo = a.first, hi = a.first + R - 1;
  if constexpr (CM != 0) {
    if (a.vmask == 0u) return 0;
    if (!(a.vmask & 1u)) lo += 1;
    if (!(a.vmask & 2u)) hi -= 1;
  }
  if constexpr (G == 2) {
    Axis<R> b;
    make_axis<MAS, CM>(g, u, 1, b);
    hi = b.first + R - 1;                        // b.first is a.first or a.first + 1
  }
  int nt = 0;
  t0 = t1 = t2 = -1;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    if (lo + k > hi) break;
    const int t = tile_of(g, ax, wrapn(lo + k, g.N));
    if (t == t0 || t == t1 || t == t2) continue;
    if (nt == 0) t0 = t; else if (nt == 1) t1 = t; else t2 = t;
    ++nt;
  }
  return nt;
}

__device__ __forceinline__ int pick3(int k, int a, int b, int c) { return k == 0 ? a : (k == 1 ? b : c); }

__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Fill path: the entries beyond a bucket's capacity.  An entry's slot is its
// rank among its bucket's attempts, so entry r of bucket b's surplus has a
// place of its own, r mod 2^lg in the chunk of key (b, r >> lg): an open hash
// table of chunks that hold particle numbers.  A tile finds any of its
// surplus entries by one probe and reads the particle from the catalogue, so
// a clump costs its own tile a few dependent loads per entry, whatever the
// number of clumps (linked lists that a few threads walked took 13.9 ms where
// this takes 4.3 for a 512^3 CIC deposit of 4 Mi particles, three quarters of
// them in 8 clumps, 7.4 against 2.4 with 20), and the table is 6 bytes per
// entry that can spill where lists and copies of the entries took 40.
struct Spill {
  unsigned long long* keys;   // [chunks], zeroed; 0: free
  unsigned* ids;              // [chunks << lg] particle numbers
  unsigned chunks;
  int lg;
};

__device__ __forceinline__ unsigned long long spill_key(const Spill& sp, unsigned bucket, unsigned rank) {
  return ((unsigned long long)(bucket + 1u) << 28) | (rank >> sp.lg);      // lg >= 4
}

__device__ __forceinline__ unsigned spill_home(const Spill& sp, unsigned long long key) {
  return (unsigned)(((key * 0x9E3779B97F4A7C15ull >> 32) * sp.chunks) >> 32);
}

// Entry `rank` of bucket `bucket`'s surplus is particle `id`.  The table has
// half as many chunks again as a catalogue can need, so a probe ends.
__device__ __forceinline__ void spill_entry(const Spill& sp, unsigned bucket, unsigned rank, unsigned id) {
  const unsigned long long key = spill_key(sp, bucket, rank);
  unsigned c = spill_home(sp, key);
  for (unsigned tries = 0; tries < sp.chunks; ++tries) {
    unsigned long long k = *const_cast<volatile unsigned long long*>(sp.keys + c);
    if (k == 0ull) {
      k = atomicCAS(sp.keys + c, 0ull, key);
      if (k == 0ull) k = key;
    }
    if (k == key) {
      sp.ids[((size_t)c << sp.lg) + (rank & ((1u << sp.lg) - 1u))] = id;
      return;
    }
    c = c + 1u == sp.chunks ? 0u : c + 1u;
  }
}

// The particle of that entry (0xffffffff should it not be there).
__device__ __forceinline__ unsigned spilled_id(const Spill& sp, unsigned bucket, unsigned rank) {
  const unsigned long long key = spill_key(sp, bucket, rank);
  unsigned c = spill_home(sp, key);
  for (unsigned tries = 0; sp.keys[c] != key; c = c + 1u == sp.chunks ? 0u : c + 1u)
    if (++tries > sp.chunks) return 0xffffffffu;
  return sp.ids[((size_t)c << sp.lg) + (rank & ((1u << sp.lg) - 1u))];
}

// A particle's entry (u, w), as the fill computed it.
__device__ __forceinline__ float4 particle_entry(const Catalogue& cat, unsigned i) {
  if (i == 0xffffffffu) return make_float4(0.f, 0.f, 0.f, 0.f);
  return make_float4(__fmul_rn(__fsub_rn(cat.x[i], cat.ox), cat.inv_cell),
                     __fmul_rn(__fsub_rn(cat.y[i], cat.oy), cat.inv_cell),
                     __fmul_rn(__fsub_rn(cat.z[i], cat.oz), cat.inv_cell), cat.w ? cat.w[i] : 1.0f);
}

// use(entry) of a tile's n spilled entries, thread by thread of NT.  A thread
// looks up the numbers of four at once and loads the next one's particle
// before it uses the last.
template <int NT, class Id, class Use>
__device__ __forceinline__ void for_spilled(const Catalogue& cat, unsigned n, Id id_of, Use use) {
  for (unsigned i0 = threadIdx.x; i0 < n; i0 += 4 * NT) {
    unsigned id[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) id[k] = i0 + k * NT < n ? id_of(i0 + k * NT) : 0xffffffffu;
    float4 e = particle_entry(cat, id[0]);
#pragma unroll 1
    for (unsigned i = i0; i < n && i < i0 + 4 * NT; i += NT) {
      const float4 next = particle_entry(cat, id[1]);
      use(e);
      e = next;
      id[1] = id[2];
      id[2] = id[3];
      id[3] = 0xffffffffu;
    }
  }
}

// The fill kernels leave the catalogue they read (the parameters' or the
// job's) beside the counters, for the tiles.
__device__ __forceinline__ void keep_catalogue(const DepGeom& g, DepCounters* ctr) {
  if (blockIdx.x == 0 && threadIdx.x == 0)
    ctr->cat = Catalogue{g.x, g.y, g.z, g.w, g.ox, g.oy, g.oz, g.inv_cell};
}

// Number of particle k of a thread's batch (load_batch).
__device__ __forceinline__ unsigned batch_id(int k) {
  return (blockIdx.x * CNT_ITEMS + k) * CNT_THREADS + threadIdx.x;
}

// Block reductions of the weight statistics in a fixed order (deterministic
// partials per particle block), and the global max |w|.
__device__ __forceinline__ void flush_block_stats(float maxw, ff sw, ff sw2, unsigned kept, unsigned bad,
                                                  DepCounters* ctr, float4* block_stats) {
  __shared__ float s_max[CNT_THREADS / 32];
  __shared__ ff s_sw[CNT_THREADS / 32], s_sw2[CNT_THREADS / 32];
  __shared__ unsigned s_kept, s_bad;
  if (threadIdx.x == 0) { s_kept = 0; s_bad = 0; }
  __syncthreads();
  maxw = warp_max(maxw);
  sw = warp_ff_sum(sw);
  sw2 = warp_ff_sum(sw2);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) { s_max[wid] = maxw; s_sw[wid] = sw; s_sw2[wid] = sw2; }
  if (kept) atomicAdd(&s_kept, kept);
  if (bad) atomicAdd(&s_bad, bad);
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = 0.f;
    ff a{0.f, 0.f}, b{0.f, 0.f};
    for (int k = 0; k < CNT_THREADS / 32; ++k) {
      m = fmaxf(m, s_max[k]);
      a = ff_add(a, s_sw[k]);
      b = ff_add(b, s_sw2[k]);
    }
    block_stats[blockIdx.x] = make_float4(a.hi, a.lo, b.hi, b.lo);
    if (s_kept) atomicAdd(&ctr->kept, (unsigned long long)s_kept);
    if (s_bad) atomicAdd(&ctr->bad, (unsigned long long)s_bad);
    if (m > 0.f) atomicMax(&ctr->maxw_bits, __float_as_uint(m));
  }
}

// Pass 1: tile occupancy counts + weight statistics.
template <int MAS, int G, int CM, bool JOB>
__global__ void __launch_bounds__(CNT_THREADS)
count_kernel(DepGeom gp, unsigned* __restrict__ counts, DepCounters* ctr, float4* block_stats) {
  pdl_wait();
  const DepGeom g = catalogue_of<JOB>(gp);
  float maxw = 0.0f;
  ff sw{0.f, 0.f}, sw2{0.f, 0.f};
  unsigned kept = 0, bad = 0;
  Batch bt;
  load_batch(g, bt, blockIdx.x);
#pragma unroll
  for (int k = 0; k < CNT_ITEMS; ++k) {
    if (!bt.in[k]) continue;
    float u[3];
    const float w = bt.w[k];
    if (!grid_coords(g, bt.x[k], bt.y[k], bt.z[k], u)) { ++bad; continue; }
    int x0, x1, x2, y0, y1, y2, z0, z1, z2;
    const int nx = axis_tiles<MAS, G, CM>(g, 0, u[0], x0, x1, x2);
    const int ny = axis_tiles<MAS, G, CM>(g, 1, u[1], y0, y1, y2);
    const int nz = axis_tiles<MAS, G, CM>(g, 2, u[2], z0, z1, z2);
    if (nx * ny * nz == 0) continue;
    ++kept;
    for (int a = 0; a < nx; ++a)
      for (int b = 0; b < ny; ++b)
        for (int c = 0; c < nz; ++c)
          atomicAdd(&counts[((pick3(a, x0, x1, x2) * g.nt[1] + pick3(b, y0, y1, y2)) * g.nt[2] +
                             pick3(c, z0, z1, z2)) * CSTRIDE], 1u);
    maxw = fmaxf(maxw, fabsf(w));
    sw = ff_add_f(sw, w);
    sw2 = ff_add_f(sw2, __fmul_rn(w, w));
  }
  flush_block_stats(maxw, sw, sw2, kept, bad, ctr, block_stats);
}

// Passes 1 and 3 at once (fill path: buckets of a fixed capacity g.tcap, tile
// t's at entry t * tcap).  The count of tile t that a particle's atomic
// returns is also its slot in t's bucket, so the entry is written right away;
// a slot beyond the capacity goes to the spill table instead, where the
// tile's CTA looks it up, so a clump costs its own tile and no second pass
// over the catalogue (a scan and a scatter that rebuilt all buckets cost 0.15
// of the 0.57 ms of a clustered 4 Mi particle 512^3 CIC deposit, and two idle
// launches when nothing overflowed).  The statistics are those of count_kernel, over the
// same particle blocks.
// Registers for 5 CTAs per SM: its returning atomics want warps in flight
// (0.151 -> 0.142 ms for 4 Mi particles at 512^3 against 4 CTAs per SM).
template <int MAS, int G, int CM, bool JOB>
__global__ void __launch_bounds__(CNT_THREADS, 5)
fill_kernel(DepGeom gp, unsigned* __restrict__ counts, float4* __restrict__ entries,
            const __grid_constant__ Spill sp, DepCounters* ctr, float4* block_stats) {
  pdl_wait();
  const DepGeom g = catalogue_of<JOB>(gp);
  keep_catalogue(g, ctr);
  const unsigned tcap = g.tcap;
  float maxw = 0.0f;
  ff sw{0.f, 0.f}, sw2{0.f, 0.f};
  unsigned kept = 0, bad = 0;
  Batch bt;
  load_batch(g, bt, blockIdx.x);
#pragma unroll
  for (int k = 0; k < CNT_ITEMS; ++k) {
    if (!bt.in[k]) continue;
    float u[3];
    const float w = bt.w[k];
    if (!grid_coords(g, bt.x[k], bt.y[k], bt.z[k], u)) { ++bad; continue; }
    int x0, x1, x2, y0, y1, y2, z0, z1, z2;
    const int nx = axis_tiles<MAS, G, CM>(g, 0, u[0], x0, x1, x2);
    const int ny = axis_tiles<MAS, G, CM>(g, 1, u[1], y0, y1, y2);
    const int nz = axis_tiles<MAS, G, CM>(g, 2, u[2], z0, z1, z2);
    if (nx * ny * nz == 0) continue;
    ++kept;
    const float4 e = make_float4(u[0], u[1], u[2], w);
    if (nx <= 2 && ny <= 2 && nz <= 2) {
      // at most 2 x 2 x 2 tiles: all slots claimed at once (the returning atomics overlap)
      int tt[8];
      unsigned slot[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int a = q >> 2, b = (q >> 1) & 1, c = q & 1;
        tt[q] = (a < nx && b < ny && c < nz)
                    ? ((a ? x1 : x0) * g.nt[1] + (b ? y1 : y0)) * g.nt[2] + (c ? z1 : z0) : -1;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (tt[q] >= 0) slot[q] = atomicAdd(&counts[tt[q] * CSTRIDE], 1u);
      bool over = false;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (tt[q] >= 0) {
          if (slot[q] < tcap) entries[(unsigned)tt[q] * tcap + slot[q]] = e;
          else over = true;
        }
      if (over) {
#pragma unroll 1
        for (int q = 0; q < 8; ++q) {
          int t = -1;
          unsigned s = 0;
#pragma unroll
          for (int r = 0; r < 8; ++r)
            if (r == q) {
              t = tt[r];
              s = slot[r];
            }
          if (t >= 0 && s >= tcap) spill_entry(sp, (unsigned)t, s - tcap, batch_id(k));
        }
      }
    } else {
      for (int a = 0; a < nx; ++a)
        for (int b = 0; b < ny; ++b)
          for (int c = 0; c < nz; ++c) {
            const int t = (pick3(a, x0, x1, x2) * g.nt[1] + pick3(b, y0, y1, y2)) * g.nt[2] + pick3(c, z0, z1, z2);
            const unsigned slot = atomicAdd(&counts[t * CSTRIDE], 1u);
            if (slot < tcap) entries[(unsigned)t * tcap + slot] = e;
            else spill_entry(sp, (unsigned)t, slot - tcap, batch_id(k));
          }
    }
    maxw = fmaxf(maxw, fabsf(w));
    sw = ff_add_f(sw, w);
    sw2 = ff_add_f(sw2, __fmul_rn(w, w));
  }
  flush_block_stats(maxw, sw, sw2, kept, bad, ctr, block_stats);
}

// Column tiles (TX x TY pencils over all of z; power-of-two meshes, TX, TY >=
// 4): a particle is written once, to the tile of its first node in x and y,
// into the part of the bucket of its class: 2 * (its nodes reach the next
// tile in x) + (in y).  A tile's entries are then nine runs (column_entries):
// its own four parts, the left neighbour's two that cross in x, the lower
// neighbour's two that cross in y, the diagonal one's that crosses in both.
// One atomic and one 16-byte store per particle instead of one per tile it
// touches (3.1 for TSC with two grids and 4x4 tiles): the returning atomics
// set this pass's time, 15 us per million (512^3, 4 Mi particles TSC, two
// grids: 0.190 -> 0.063 ms; 256^3, 1 M: 0.047 -> 0.022; 1024^3, 16 Mi PCS:
// 1.28 -> 0.32), for 2 % more in the kernel that finds the runs.
constexpr int CLS = CSTRIDE / 4;              // words between a tile's four class counters (a sector each)

// v[c] by selects (no local memory).
__device__ __forceinline__ unsigned pick4(unsigned c, const unsigned (&v)[4]) {
  return (c & 2u) ? ((c & 1u) ? v[3] : v[2]) : ((c & 1u) ? v[1] : v[0]);
}

template <int MAS, int G>
__device__ __forceinline__ int column_axis(const DepGeom& g, int ax, float u, int& cross) {
  Axis<MAS> a;
  make_axis<MAS, 0>(g, u, 0, a);
  int last = a.first + MAS - 1;
  if constexpr (G == 2) {
    Axis<MAS> b;
    make_axis<MAS, 0>(g, u, 1, b);
    last = b.first + MAS - 1;                 // b.first is a.first or a.first + 1
  }
  const int f = a.first & (g.N - 1);
  cross = (f & (g.td[ax] - 1)) + (last - a.first) >= g.td[ax] ? 1 : 0;
  return f >> g.ts[ax];
}

template <int MAS, int G, bool JOB>
__global__ void __launch_bounds__(CNT_THREADS, 5)
fill_columns_kernel(DepGeom gp, unsigned* __restrict__ counts, float4* __restrict__ entries,
                    const __grid_constant__ Spill sp, DepCounters* ctr, float4* block_stats) {
  pdl_wait();
  const DepGeom g = catalogue_of<JOB>(gp);
  keep_catalogue(g, ctr);
  float maxw = 0.0f;
  ff sw{0.f, 0.f}, sw2{0.f, 0.f};
  unsigned kept = 0, bad = 0;
  Batch bt;
  load_batch(g, bt, blockIdx.x);
  float4 e[CNT_ITEMS];
  int tc[CNT_ITEMS];                          // 4 * tile + class, -1: dropped
  unsigned slot[CNT_ITEMS];
#pragma unroll
  for (int k = 0; k < CNT_ITEMS; ++k) {       // every particle's claim in flight before the first store
    tc[k] = -1;
    if (!bt.in[k]) continue;
    float u[3];
    const float w = bt.w[k];
    if (!grid_coords(g, bt.x[k], bt.y[k], bt.z[k], u)) { ++bad; continue; }
    int cx, cy;
    const int tx = column_axis<MAS, G>(g, 0, u[0], cx), ty = column_axis<MAS, G>(g, 1, u[1], cy);
    ++kept;
    e[k] = make_float4(u[0], u[1], u[2], w);
    const int t = tx * g.nt[1] + ty, c = 2 * cx + cy;
    tc[k] = 4 * t + c;
    slot[k] = atomicAdd(&counts[(size_t)t * CSTRIDE + c * CLS], 1u);
    maxw = fmaxf(maxw, fabsf(w));
    sw = ff_add_f(sw, w);
    sw2 = ff_add_f(sw2, __fmul_rn(w, w));
  }
  bool over = false;
#pragma unroll
  for (int k = 0; k < CNT_ITEMS; ++k) {
    if (tc[k] < 0) continue;
    const unsigned t = (unsigned)tc[k] >> 2, c = (unsigned)tc[k] & 3u;
    if (slot[k] < pick4(c, g.ccap)) entries[(size_t)t * g.tcap + pick4(c, g.coff) + slot[k]] = e[k];
    else over = true;
  }
  if (over) {                                 // a loop: in line twice, it cost the others 2-4 % of the pass
    static_assert(CNT_ITEMS == 2, "selects of two");
#pragma unroll 1
    for (int k = 0; k < CNT_ITEMS; ++k) {
      const int b = k ? tc[1] : tc[0];
      const unsigned s = k ? slot[1] : slot[0], cap = pick4((unsigned)b & 3u, g.ccap);
      if (b >= 0 && s >= cap) spill_entry(sp, (unsigned)b, s - cap, batch_id(k));
    }
  }
  flush_block_stats(maxw, sw, sw2, kept, bad, ctr, block_stats);
}

// The nine runs of a column tile's entries: entry i of the buckets lies at
// i + delta[r], r the last run with pre[r] <= i (runs 9.. never are).
struct ColRuns {
  unsigned pre[16], delta[16];
  unsigned spilled[9], code[9];               // entries beyond the bucket, 4 * tile + class
  unsigned total, n_spilled;
};

struct ColEntries {
  const float4* entries;
  const ColRuns* runs;
  const Spill* sp;
  const DepCounters* ctr;
  unsigned n[2];                              // in buckets, spilled
};

// Where entry i of the buckets lies.
__device__ __forceinline__ unsigned column_index(const ColEntries& te, unsigned i) {
  const ColRuns& r = *te.runs;
  int q = i >= r.pre[8] ? 8 : 0;
  if (i >= r.pre[q + 4]) q += 4;
  if (i >= r.pre[q + 2]) q += 2;
  if (i >= r.pre[q + 1]) q += 1;
  return i + r.delta[q];
}

// The particle of spilled entry i of a column tile.
__device__ __forceinline__ unsigned spilled_column(const ColEntries& te, unsigned i) {
  const ColRuns& r = *te.runs;
  int q = 0;
  while (q < 8 && i >= r.spilled[q]) i -= r.spilled[q++];
  return spilled_id(*te.sp, r.code[q], i);
}

// Every thread of the block calls; ends with a barrier.
__device__ __forceinline__ ColEntries column_entries(const DepGeom& g, int tx, int ty, const float4* entries,
                                                     const unsigned* counts, const Spill& sp,
                                                     const DepCounters* ctr, ColRuns& r) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    unsigned m = 0, code = 0, c = 0;
    if (lane < 9) {
      // own 0..3 | left, crossing in x: 2, 3 | lower, crossing in y: 1, 3 | diagonal: 3
      const int dx = (lane == 4 || lane == 5 || lane == 8) ? 1 : 0, dy = lane >= 6 ? 1 : 0;
      const int cls = lane < 4 ? lane : (lane == 4 ? 2 : (lane == 6 ? 1 : 3));
      const int ntx = g.nt[0], nty = g.nt[1];
      const int t = ((tx + ntx - dx) & (ntx - 1)) * nty + ((ty + nty - dy) & (nty - 1));
      code = 4u * t + cls;
      c = counts[(size_t)t * CSTRIDE + cls * CLS];
      m = min(c, g.ccap[cls]);
    }
    unsigned inc = m;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    const unsigned all = __reduce_add_sync(0xffffffffu, c - m);
    if (lane < 16) {
      const unsigned first = lane < 9 ? (code >> 2) * g.tcap + g.coff[code & 3u] : 0u;
      r.pre[lane] = lane < 9 ? inc - m : 0xffffffffu;
      r.delta[lane] = first - (inc - m);
      if (lane < 9) {
        r.spilled[lane] = c - m;
        r.code[lane] = code;
      }
      if (lane == 8) r.total = inc;
      if (lane == 0) r.n_spilled = all;
    }
  }
  __syncthreads();
  ColEntries te;
  te.entries = entries;
  te.runs = &r;
  te.sp = &sp;
  te.ctr = ctr;
  te.n[0] = r.total;
  te.n[1] = r.n_spilled;
  return te;
}

// The entries of one tile in two parts: n[0] in its bucket, n[1] beyond its
// capacity (fill path).  A tile that has any of the rare second part goes
// through a copy of its code out of line: a call, or a second loop, in the
// common one would cost it registers (512^3 CIC, 4 Mi particles: 279 -> 387 us
// with the call in the middle).
struct TileEntries {
  const float4* entries;
  const Spill* sp;
  const DepCounters* ctr;
  unsigned t, n[2];
};

__device__ __forceinline__ TileEntries tile_entries(const DepGeom& g, int t, const float4* entries,
                                                    const unsigned* counts, const unsigned* offsets, const Spill& sp,
                                                    const DepCounters* ctr) {
  TileEntries te;
  const unsigned c = counts[(long long)t * CSTRIDE];
  te.entries = entries + (g.tcap ? (size_t)t * g.tcap : (size_t)offsets[t]);
  te.sp = &sp;
  te.ctr = ctr;
  te.t = (unsigned)t;
  te.n[0] = g.tcap ? min(c, g.tcap) : c;
  te.n[1] = c - te.n[0];
  return te;
}

// Pass 3: append (u_x, u_y, u_z, w) to every touched tile's bucket.
template <int MAS, int G, int CM, bool JOB>
__global__ void __launch_bounds__(CNT_THREADS, 4)
scatter_kernel(DepGeom gp, const unsigned* __restrict__ offsets, unsigned* __restrict__ fills,
               float4* __restrict__ entries) {
  pdl_wait();
  const DepGeom g = catalogue_of<JOB>(gp);
  {
    Batch bt;
    load_batch(g, bt, blockIdx.x);
#pragma unroll
    for (int k = 0; k < CNT_ITEMS; ++k) {
      if (!bt.in[k]) continue;
      float u[3];
      const float w = bt.w[k];
      if (!grid_coords(g, bt.x[k], bt.y[k], bt.z[k], u)) continue;
      int x0, x1, x2, y0, y1, y2, z0, z1, z2;
      const int nx = axis_tiles<MAS, G, CM>(g, 0, u[0], x0, x1, x2);
      const int ny = axis_tiles<MAS, G, CM>(g, 1, u[1], y0, y1, y2);
      const int nz = axis_tiles<MAS, G, CM>(g, 2, u[2], z0, z1, z2);
      if (nx * ny * nz == 0) continue;
      const float4 e = make_float4(u[0], u[1], u[2], w);
      if (nx <= 2 && ny <= 2 && nz <= 2) {
        // at most 2 x 2 x 2 tiles (every tile at least as wide as the stencil): all slots claimed at
        // once, so the returning atomics of one particle overlap instead of forming a chain
        int tt[8];
        unsigned base[8], slot[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int a = q >> 2, b = (q >> 1) & 1, c = q & 1;
          tt[q] = (a < nx && b < ny && c < nz)
                      ? ((a ? x1 : x0) * g.nt[1] + (b ? y1 : y0)) * g.nt[2] + (c ? z1 : z0) : -1;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (tt[q] >= 0) {
            base[q] = offsets[tt[q]];
            slot[q] = atomicAdd(&fills[tt[q] * CSTRIDE], 1u);
          }
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (tt[q] >= 0) entries[base[q] + slot[q]] = e;
      } else {
        for (int a = 0; a < nx; ++a)
          for (int b = 0; b < ny; ++b)
            for (int c = 0; c < nz; ++c) {
              const int t = (pick3(a, x0, x1, x2) * g.nt[1] + pick3(b, y0, y1, y2)) * g.nt[2] + pick3(c, z0, z1, z2);
              entries[offsets[t] + atomicAdd(&fills[t * CSTRIDE], 1u)] = e;
            }
      }
    }
  }
}

// int64 fixed-point value -> float32 (two exact 32-bit halves, one rounding in the FMA).
__device__ __forceinline__ float fixed_to_float(long long q, float inv_sc) {
  const int hi = (int)(q >> 32);
  const unsigned lo = (unsigned)(q & 0xffffffffull);
  const float v = __fmaf_rn(__int2float_rn(hi), 4294967296.0f, __uint2float_rn(lo));
  return __fmul_rn(v, inv_sc);
}

// Local (in-tile) coordinate of stencil node r of an axis, or -1.
template <int R>
__device__ __forceinline__ void local_nodes(const Axis<R>& a, int N, int t0, int ext, int (&l)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int c = wrapn(a.first + r, N) - t0;
    l[r] = (((a.vmask >> r) & 1u) && c >= 0 && c < ext) ? c : -1;
  }
}

// Pass 5 of the mesh deposit: gbp_deposit_stats from the counters and the
// per-block partials (the fused path folds them in power_reduce_kernel).
__global__ void __launch_bounds__(STATS_LANES)
stats_kernel(StatsFold f) {
  pdl_wait();
  fold_stats<STATS_LANES>(f);
}

struct DepLayout {
  int td[3], ts[3], nt[3], ntiles, maxrep, nblocks;
  unsigned tcap;        // fill path: entries per bucket (0: count path)
  unsigned flag_cap;    // DepGeom::flag_cap
  unsigned ccap[4], coff[4];   // column tiles: each class's part of the bucket
  size_t nentries;      // entries the bucket buffer holds
  size_t chunks;        // fill path: chunks of 2^lg entries of the spill table
  int lg;
  size_t scan_bytes;
  size_t total;
};

// Bytes at the start of the workspace that one memset clears per call: the
// counters, the tiles' entry counts and their fill counters or the spill
// table's keys (adjacent).
inline size_t zeroed_bytes(const DepLayout& L) {
  const size_t counts = align256((size_t)L.ntiles * CSTRIDE * sizeof(unsigned));
  return align256(sizeof(DepCounters)) + counts + (L.tcap ? align256(L.chunks * sizeof(unsigned long long)) : counts);
}

struct StrideLoad {
  const unsigned* p;
  __host__ __device__ unsigned operator()(int i) const { return p[(long long)i * CSTRIDE]; }
};

inline thrust::transform_iterator<StrideLoad, thrust::counting_iterator<int>> strided_counts(const unsigned* p) {
  return thrust::make_transform_iterator(thrust::counting_iterator<int>(0), StrideLoad{p});
}

void finish_layout(DepLayout& L);

// Spill table of `nlists` buckets whose surplus is at most `most` entries:
// chunks of about a bucket's mean fill (16 to 128 entries, so that neither
// part-filled chunks nor keys take much), half as many again as can be in use
// (every full one, and a part-filled one per bucket).
void size_spill(DepLayout& L, double most, double nlists) {
  L.lg = 4;
  while (L.lg < 7 && most / nlists > (double)(1 << L.lg)) ++L.lg;
  L.chunks = (size_t)(1.5 * std::min(most, nlists + most / (double)(1 << L.lg))) + 16;
}

// Mean entries per tile of a uniform catalogue of n particles (a span of
// `width` nodes reaches the next tile along an axis with probability
// (width - 1) / td), and the capacity of a bucket for it.
double mean_fill(int64_t n, int N, int width, const DepLayout& L) {
  double rep = 1.0;
  for (int a = 0; a < 3; ++a)
    if (L.td[a] < N) rep *= 1.0 + (double)(width - 1) / (double)L.td[a];
  return (double)n * rep / (double)L.ntiles;
}
double bucket_capacity(double mean) { return 4.0 * std::ceil((2.0 * mean + 64.0) / 4.0); }

// Largest number of distinct tiles a run of `width` consecutive nodes can
// touch along one periodic axis (exact, by enumeration).
int max_tiles_axis(int N, int tdim, int width) {
  int best = 0;
  for (int s = 0; s < N; ++s) {
    int seen[8], ns = 0;
    for (int r = 0; r < width; ++r) {
      const int t = ((s + r) % N) / tdim;
      bool dup = false;
      for (int k = 0; k < ns; ++k) dup = dup || seen[k] == t;
      if (!dup && ns < 8) seen[ns++] = t;
    }
    best = ns > best ? ns : best;
  }
  return best;
}

// Tiles of td[0] x td[1] x td[2] cells (each at most N); every particle goes
// to the bucket of each tile its stencil (all grids) touches.  fill: buckets
// of a fixed capacity, twice the mean fill m of a uniform catalogue of n
// particles plus 64 (a span of `width` nodes reaches the next tile along an
// axis with probability (width - 1) / td), so that spills are rare unless the
// catalogue is strongly clustered; the count path when m < 32 and the buckets
// would still take more than 256 MB (a large mesh with few particles).  Wider
// buckets cost the one pass time: the same entries written over a larger
// range (3 m + 64 instead of 2 m + 64: 0.169 against 0.147 ms for 4 Mi
// particles at 512^3).
int deposit_layout(int64_t n, int N, int mas, int interlace, int compat, const int (&tile)[3], DepLayout& L,
                   bool fill = false) {
  if (N < 1 || N > 4096) return GBP_ERR_INVALID;
  if (n < 0) return GBP_ERR_INVALID;
  if (mas < GBP_NGP || mas > GBP_PCS) return GBP_ERR_INVALID;
  if (compat < 0 || compat > GBP_COMPAT_SCAN) return GBP_ERR_INVALID;
  if (compat && (mas != GBP_CIC || interlace)) return GBP_ERR_INVALID;
  const int R = compat ? 2 : mas;
  const int width = R + (interlace ? 1 : 0);
  L.ntiles = 1;
  L.maxrep = 1;
  for (int a = 0; a < 3; ++a) {
    L.td[a] = N < tile[a] ? N : tile[a];
    L.ts[a] = (L.td[a] & (L.td[a] - 1)) == 0 ? __builtin_ctz(L.td[a]) : -1;
    L.nt[a] = (N + L.td[a] - 1) / L.td[a];
    const int m = max_tiles_axis(N, L.td[a], width);
    if (m > 3) return GBP_ERR_UNSUPPORTED;
    L.ntiles *= L.nt[a];
    L.maxrep *= m;
  }
  if ((double)n * L.maxrep >= 4294967295.0) return GBP_ERR_UNSUPPORTED;
  L.nblocks = (int)((n + (long long)CNT_THREADS * CNT_ITEMS - 1) / ((long long)CNT_THREADS * CNT_ITEMS));
  L.tcap = 0;
  L.nentries = (size_t)n * L.maxrep + 1;
  L.chunks = 0;
  L.lg = 4;
  L.flag_cap = 0xffffffffu;
  if (fill && n > 0) {
    const double mean = mean_fill(n, N, width, L), cap = bucket_capacity(mean);
    if (mean >= 32.0) L.flag_cap = (unsigned)std::min(cap, 4294967295.0);
    if ((mean >= 32.0 || cap * (double)L.ntiles <= 16777216.0) && cap * (double)L.ntiles < 4294967295.0) {
      L.tcap = (unsigned)cap;
      size_spill(L, (double)n * L.maxrep, L.ntiles);
      L.nentries = (size_t)L.tcap * (size_t)L.ntiles + 1;
    }
  }
  finish_layout(L);
  return GBP_OK;
}

// Column tiles of tx x ty pencils (both powers of two >= 4 that divide N/2),
// always one pass: class c's part of a bucket holds twice its mean fill of a
// uniform catalogue plus 48 (what overflows it goes to the spill table;
// GBP_STATS_REFILLED is reported at the capacity a bucket of all the tile's
// entries would have).  Nodes first .. last of all grids span MAS - 1 cells,
// or half a cell more on average with two grids, so they reach the next tile
// along an axis with probability span / tx.
int column_layout(int64_t n, int N, int mas, int interlace, int tx, int ty, DepLayout& L) {
  if (n < 0) return GBP_ERR_INVALID;
  if (mas < GBP_NGP || mas > GBP_PCS) return GBP_ERR_INVALID;
  const int td[3] = {tx, ty, N}, width = mas + (interlace ? 1 : 0);
  L.maxrep = 1;
  for (int a = 0; a < 3; ++a) {
    L.td[a] = td[a];
    L.ts[a] = __builtin_ctz(td[a]);
    L.nt[a] = N / td[a];
    // tiles that `width` consecutive nodes can touch (td divides N): no enumeration in a call's host time
    if (a < 2) L.maxrep *= std::min(L.nt[a], 1 + (width + td[a] - 2) / td[a]);
  }
  L.ntiles = L.nt[0] * L.nt[1];
  if ((double)n * L.maxrep >= 4294967295.0) return GBP_ERR_UNSUPPORTED;
  L.nblocks = (int)((n + (long long)CNT_THREADS * CNT_ITEMS - 1) / ((long long)CNT_THREADS * CNT_ITEMS));
  const double all = mean_fill(n, N, width, L);
  L.flag_cap = all >= 32.0 ? (unsigned)std::min(bucket_capacity(all), 4294967295.0) : 0xffffffffu;
  const double span = mas - 1 + (interlace ? 0.5 : 0.0), mean = (double)n / (double)L.ntiles;
  // entries are numbered in 32 bits: less than twice the mean beyond 2.1e9 particles (NGP on one grid, whose
  // particles touch one tile, takes up to 4.29e9), the surplus in the table
  const double slack = 4.0 * 52.0 * (double)L.ntiles;
  const double f = n > 0 ? std::min(2.0, (4294967295.0 - slack) / (double)n) : 2.0;
  double off = 0.0;
  for (int c = 0; c < 4; ++c) {
    const double px = span / tx, py = span / ty;
    const double m = mean * ((c & 2) ? px : 1.0 - px) * ((c & 1) ? py : 1.0 - py);
    const double cap = 4.0 * std::ceil((f * m + 48.0) / 4.0);
    L.coff[c] = (unsigned)off;
    L.ccap[c] = (unsigned)cap;
    off += cap;
  }
  L.tcap = (unsigned)off;
  L.nentries = (size_t)L.tcap * (size_t)L.ntiles + 1;
  size_spill(L, (double)n, 4.0 * L.ntiles);
  finish_layout(L);
  return GBP_OK;
}

// The rest of a layout, from its tiles, blocks and buckets.
void finish_layout(DepLayout& L) {
  L.scan_bytes = 0;
  if (!L.tcap)
    cub::DeviceScan::ExclusiveSum(nullptr, L.scan_bytes, strided_counts(nullptr), (unsigned*)nullptr, L.ntiles);
  const size_t nbl = (size_t)(L.nblocks > 0 ? L.nblocks : 1);
  L.total = zeroed_bytes(L) + align256((size_t)L.ntiles * 2 * sizeof(long long)) + align256((size_t)L.ntiles * 4) +
            align256(nbl * sizeof(float4)) +
            align256(L.nentries * sizeof(float4)) + align256(L.scan_bytes) +
            align256((L.chunks << L.lg) * sizeof(unsigned));
}

// Workspace slices shared by both deposit paths.
struct DepBuffers {
  DepCounters* ctr;
  unsigned* counts;      // [ntiles * CSTRIDE] entries per tile (count pass)
  unsigned* fills;       // [ntiles * CSTRIDE] entries written so far (count path's scatter; else nullptr)
  unsigned* offsets;     // [ntiles] first entry of each tile (exclusive scan of the counts)
  float4* block_stats;
  long long* tile_mass;  // [2][ntiles]
  float4* entries;
  void* scan_tmp;
  Spill spill;           // fill path
};

inline DepBuffers carve_deposit(void* workspace, const DepLayout& L) {
  Carver cv(workspace);
  DepBuffers b;
  const int nbl = L.nblocks > 0 ? L.nblocks : 1;
  b.ctr = cv.take<DepCounters>(1);
  b.counts = cv.take<unsigned>((size_t)L.ntiles * CSTRIDE);
  b.fills = L.tcap ? nullptr : cv.take<unsigned>((size_t)L.ntiles * CSTRIDE);
  b.spill.keys = L.tcap ? cv.take<unsigned long long>(L.chunks) : nullptr;
  b.offsets = cv.take<unsigned>(L.ntiles);
  b.block_stats = cv.take<float4>(nbl);
  b.tile_mass = cv.take<long long>((size_t)L.ntiles * 2);
  b.entries = cv.take<float4>(L.nentries);
  b.scan_tmp = cv.take<char>(L.scan_bytes);
  b.spill.ids = cv.take<unsigned>(L.chunks << L.lg);
  b.spill.chunks = (unsigned)L.chunks;
  b.spill.lg = L.lg;
  return b;
}

// Passes 1-3: bucket the particles by tile (the first zeroed_bytes(L) of the
// workspace must be zero on entry).
template <int MAS, int G, int CM>
int bucket_particles(const DepGeom& g, const DepLayout& L, const DepBuffers& b, cudaStream_t st) {
  const bool job = g.job != nullptr;                 // B-spline deposits only
  if (L.tcap) {
    if (L.nblocks > 0) {
      GBP_TRACE("deposit_fill", st);
      GBP_CUDA_TRY(launch_pdl(job ? fill_kernel<MAS, G, CM, CM == 0> : fill_kernel<MAS, G, CM, false>,
                              dim3(L.nblocks), dim3(CNT_THREADS), 0, st, g, b.counts, b.entries, b.spill, b.ctr,
                              b.block_stats));
    }
    return GBP_OK;
  }
  if (L.nblocks > 0) {
    GBP_TRACE("deposit_count", st);
    GBP_CUDA_TRY(launch_pdl(job ? count_kernel<MAS, G, CM, CM == 0> : count_kernel<MAS, G, CM, false>,
                            dim3(L.nblocks), dim3(CNT_THREADS), 0, st, g, b.counts, b.ctr, b.block_stats));
  }
  {
    GBP_TRACE("deposit_scan", st);
    size_t scan_bytes = L.scan_bytes;
    GBP_CUDA_TRY(cub::DeviceScan::ExclusiveSum(b.scan_tmp, scan_bytes, strided_counts(b.counts), b.offsets,
                                               L.ntiles, st));
  }
  if (L.nblocks > 0) {
    GBP_TRACE("deposit_scatter", st);
    GBP_CUDA_TRY(launch_pdl(job ? scatter_kernel<MAS, G, CM, CM == 0> : scatter_kernel<MAS, G, CM, false>,
                            dim3(L.nblocks), dim3(CNT_THREADS), 0, st, g, b.offsets, b.fills, b.entries));
  }
  return GBP_OK;
}

// The same for column tiles.
template <int MAS, int G>
int bucket_columns(const DepGeom& g, const DepLayout& L, const DepBuffers& b, cudaStream_t st) {
  if (L.nblocks == 0) return GBP_OK;
  GBP_TRACE("deposit_fill", st);
  auto k = g.job ? fill_columns_kernel<MAS, G, true> : fill_columns_kernel<MAS, G, false>;
  GBP_CUDA_TRY(launch_pdl(k, dim3(L.nblocks), dim3(CNT_THREADS), 0, st, g, b.counts,
                          b.entries, b.spill, b.ctr, b.block_stats));
  return GBP_OK;
}

inline StatsFold stats_fold(const DepBuffers& b, const DepLayout& L, int compat, int G, gbp_deposit_stats* out) {
  return StatsFold{b.ctr, b.block_stats, L.nblocks, compat, G, b.tile_mass, L.ntiles, out};
}

inline int deposit_stats(const DepBuffers& b, const DepLayout& L, int compat, int G, gbp_deposit_stats* out,
                         cudaStream_t st) {
  GBP_TRACE("deposit_stats", st);
  GBP_CUDA_TRY(launch_pdl(stats_kernel, dim3(1), dim3(STATS_LANES), 0, st, stats_fold(b, L, compat, G, out)));
  return GBP_OK;
}

}  // namespace
}  // namespace gbp
