// Particles -> multipole sums with the deposit fused into the z pass of the
// FFT (library transform sizes: power-of-two meshes 64..1024, B-spline
// deposits).  Included by one translation unit per mesh size
// (depfft_n<N>.cu); depfft.cu holds the C ABI and picks the unit by N.
//
// The mesh is never written.  Particles are bucketed (deposit_core.cuh) by
// column tile: TX x TY pencils spanning the whole z axis (the tile shape is
// a plan option: 4x4, 8x4 or 8x8, see column_tile_variants), each in the tile
// of its first node, by which faces its stencil crosses.  One CTA per column
// tile reads its own bucket and the crossing parts of three neighbours':
//
//   1. accumulates its bucket in shared memory as 32-bit fixed point.  Each
//      4x4-pencil block of the tile has a scale of its own, 2^s with
//      s = s_g - ceil(log2(c)) (+1 for TSC and PCS, whose node weights stay
//      below 1/2), where c is the largest number of entries that cover the
//      block in one z plane (counted first) and 2^s_g puts the largest
//      particle weight just below 2^30.  No cell can then exceed 2^30 +
//      rounding in magnitude, whatever the order of the adds, so the integer
//      sums are exact, order-independent and overflow-free (fire-and-forget
//      shared reductions, no carries).  The scales belong to the 4x4 blocks,
//      not to the tile, so every tile shape gives the same cells, the same
//      floats and the same P_l, bit for bit;
//   2. transforms its pencils along z in the packed layout (fft.cu): a complex
//      column is a pencil of both grids, or with one grid two pencils of
//      adjacent x planes.  The first radix-8 stage reads the integer cells,
//      converts them to float and writes the complex buffer that aliases the
//      accumulators; the stages in between run in place (fft_pass.cuh),
//   3. stores Z(kz) and Z(-kz) from the last stage's registers,
//   4. adds up the tile's exact integer total at the common scale 2^s_g
//      (the mean density).
//
// A tile is taken in units whose cells, all grids', fit in shared memory
// together: the tile itself where they do (UNIT_BYTES), else 4x4 pencils.
//
// A block whose densest plane would cost more than SH_MAX bits (a dense
// clump) makes its whole tile wide: 64-bit cells (the unit's on the smallest
// meshes, else half a unit at a time in the same shared memory), the clumped
// blocks at the common scale, the others at their own.  A tile with entries
// beyond its bucket's capacity takes a copy of the code out of line that looks
// them up too.
//
// Then the y pass (fft.cu) and the x pass fused with the binning (xbin.cu)
// finish the transform and the P_l sums.  HBM traffic per grid: the
// spectrum is written once here, read and written by the y pass, and read
// once by the binning; no mesh goes through HBM.
#pragma once

#include <algorithm>
#include <type_traits>

#include "deposit_core.cuh"
#include "fft_pass.cuh"
#include "gbp_bins.h"
#include "gbp_fft.h"

namespace gbp {
namespace {

template <int N, int TX_, int TY_>
struct ColTile {
  static constexpr int TX = TX_, TY = TY_;
  static constexpr int SBX = TX / 4, SBY = TY / 4, NSB = SBX * SBY;    // 4x4-pencil scale blocks
  static_assert(TX % 4 == 0 && TY % 4 == 0, "tiles are whole 4x4 scale blocks");
};

// The pencils of a tile that go through shared memory together, as PAIRS
// packed complex columns: column q = (a, ly) with a = the pencil's x (two
// grids) or x / 2 (one grid), a = q / UY, ly = q % UY.  Columns 2cp and
// 2cp + 1 always lie in one scale block.  The unit is the tile where its
// cells fit UNIT_BYTES, else 4x4 pencils of it; with 64-bit cells the same on
// the smallest meshes, else half of that or less.  At 512^3 a unit of 64 KB (512 threads, 64-thread named
// barriers, two CTAs per SM) beats one of 128 KB in a 1024-thread CTA (0.84
// against 0.89 ms for 8x4 tiles of two grids, 4 Mi particles TSC); at 1024^3
// 4x4 pencils in one CTA beat two visits of the bucket by 4x2 (7.7 against
// 8.5 ms, 16 Mi PCS).
template <int N>
constexpr size_t UNIT_BYTES = (N == 512 ? 64 : 128) * 1024;

template <int N, int G, class CT, bool WIDE>
struct Unit {
  static constexpr size_t PENCIL = (size_t)N * G * sizeof(int);          // bytes of a pencil's 32-bit cells
  static constexpr bool WHOLE = CT::TX * CT::TY * PENCIL <= UNIT_BYTES<N>;
  static constexpr int NARROW_X = WHOLE ? CT::TX : 4, NARROW_Y = WHOLE ? CT::TY : 4;
  // threads of the CTA: a butterfly pair (two columns) of the 32-bit unit's radix-8 stages each
  static constexpr int NFFT = NARROW_X * NARROW_Y * G * N / 32;
  static constexpr int NT = NFFT < 256 ? 256 : NFFT;
  // 64 registers a thread for every size: the kernel waits at the barriers between its phases, and a fourth
  // block of 256 threads hides them (256^3 TSC weighted 253 -> 244 us a call, 24 mocks of 128^3 1543 -> 1446)
  static constexpr int MINB = NT >= 1024 ? 1 : (NT >= 512 ? 2 : 4);   // CTAs per SM the registers are sized for
  static constexpr int LIST = 4 * NT;              // entries whose places are kept between the two passes
  // ints beside the cells: plane counts, list
  static constexpr size_t REST = (size_t)CT::NSB * N + LIST;
  // 64-bit cells of the whole 32-bit unit where they take 16 KB, so that a dense clump's entries are visited once
  // (64^3 TSC on one grid, 8 clumps of 9,000: 1.42 -> 1.24 ms; 128^3 CIC on one grid, 8 of 98,000: 10.1 -> 6.0);
  // 32 KB would speed up clumps at 128^3 with two grids too (11.3 -> 8.2 ms) but cost ordinary mocks in lanes 2 %
  static constexpr size_t NARROW_BYTES = NARROW_X * NARROW_Y * PENCIL;
  static constexpr bool WIDE_WHOLE = 2 * NARROW_BYTES <= 16 * 1024;
  static constexpr int UX = WIDE && !WIDE_WHOLE ? 4 : NARROW_X;
  static constexpr int UY = WIDE && !WIDE_WHOLE ? (NARROW_X * NARROW_Y == 16 ? 2 : 4) : NARROW_Y;
  static constexpr int NUY = CT::TY / UY, NU = (CT::TX / UX) * NUY;      // units per tile
  static constexpr int PAIRS = UX * UY * G / 2;
  static constexpr int SBY = UY >= 4 ? UY / 4 : 1, NSB = UX / 4 * SBY;   // scale blocks it spans
  static constexpr size_t CELLS = (size_t)2 * PAIRS * N;
  static constexpr size_t ROOM = NARROW_BYTES / sizeof(int) * (WIDE_WHOLE ? 2 : 1);     // ints the cells may take
  static constexpr size_t SMEM = (ROOM + REST) * sizeof(int);
  static_assert(CELLS * (WIDE ? 2 : 1) <= ROOM && NT <= 1024, "the unit's cells fit");
  // First cell of pencil (lx, ly) of a grid.
  __device__ static __forceinline__ int cell_row(int lx, int ly, int grid) {
    if constexpr (G == 2) return ((lx * UY + ly) * 2 + grid) * N;
    else return (((lx >> 1) * UY + ly) * 2 + (lx & 1)) * N;
  }
};

// v[b] for a block index known only at run time, by selects (no local memory).
template <int NSB, class T>
__device__ __forceinline__ T pick_block(int b, const T (&v)[NSB]) {
  T r = v[0];
#pragma unroll
  for (int k = 1; k < NSB; ++k) r = b == k ? v[k] : r;
  return r;
}

// Sum over the warp, in every lane: three 26-bit parts (12 signed bits in the
// last), each summed in 32 bits without overflow.
__device__ __forceinline__ long long warp_sum(long long v) {
  const unsigned lo = __reduce_add_sync(0xffffffffu, (unsigned)v & 0x3ffffffu);
  const unsigned mid = __reduce_add_sync(0xffffffffu, (unsigned)(v >> 26) & 0x3ffffffu);
  const int hi = __reduce_add_sync(0xffffffffu, (int)(v >> 52));
  return (long long)lo + ((long long)mid << 26) + (long long)((unsigned long long)(long long)hi << 52);
}

// Bits of resolution a block may give up to its 32-bit cells.  A block whose
// densest z plane is covered by more than 2^(SH_MAX + WBIT) entries (a dense
// clump: a halo, a point mass) is deposited with 64-bit cells at the common
// scale instead: with the coarse quantum the rounding of many identical
// contributions adds up instead of averaging out.
constexpr int SH_MAX = 10;

template <int N, int G, class CT, bool WIDE>
using UnitCell = typename std::conditional<WIDE, unsigned long long, int>::type;

// Adds entry e (all grids) to the cells of the unit at (x0, y0); up: 2^s of
// its scale blocks.
template <int N, int MAS, int G, class CT, bool WIDE>
__device__ __forceinline__ void add_entry(const DepGeom& g, const float4& e,
                                          const float (&up)[Unit<N, G, CT, WIDE>::NSB], int x0, int y0,
                                          UnitCell<N, G, CT, WIDE>* acc) {
  using U = Unit<N, G, CT, WIDE>;
  constexpr int R = MAS, UX = U::UX, UY = U::UY, NSB = U::NSB, SBY = U::SBY;
#pragma unroll
  for (int grid = 0; grid < G; ++grid) {
    Axis<R> ax, ay, az;
    make_axis<MAS, 0, N>(g, e.x, grid, ax);
    make_axis<MAS, 0, N>(g, e.y, grid, ay);
    make_axis<MAS, 0, N>(g, e.z, grid, az);
    int lx[R], ly[R], zz[R];
    local_nodes<R>(ax, N, x0, UX, lx);
    local_nodes<R>(ay, N, y0, UY, ly);
    // z weight times the particle weight at each block's scale (exact: powers of two)
    float wz[NSB][R];
#pragma unroll
    for (int r = 0; r < R; ++r) zz[r] = wrapn(az.first + r, N);
#pragma unroll
    for (int b = 0; b < NSB; ++b) {
      const float wsc = __fmul_rn(e.w, up[b]);
#pragma unroll
      for (int r = 0; r < R; ++r) wz[b][r] = __fmul_rn(az.w[r], wsc);
    }
#pragma unroll
    for (int rx = 0; rx < R; ++rx) {
      if (lx[rx] < 0) continue;
      // with one block row the block depends on x only: select the z weights once per x node
      float wzx[R];
      if constexpr (SBY == 1) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float wzb[NSB];
#pragma unroll
          for (int k = 0; k < NSB; ++k) wzb[k] = wz[k][r];
          wzx[r] = pick_block<NSB>(lx[rx] >> 2, wzb);
        }
      }
#pragma unroll
      for (int ry = 0; ry < R; ++ry) {
        if (ly[ry] < 0) continue;
        const float wxy = __fmul_rn(ax.w[rx], ay.w[ry]);
        const int row = U::cell_row(lx[rx], ly[ry], grid);
#pragma unroll
        for (int rz = 0; rz < R; ++rz) {
          float wzr;
          if constexpr (SBY == 1) {
            wzr = wzx[rz];
          } else {
            float wzb[NSB];
#pragma unroll
            for (int k = 0; k < NSB; ++k) wzb[k] = wz[k][rz];
            wzr = pick_block<NSB>((lx[rx] >> 2) * SBY + (ly[ry] >> 2), wzb);
          }
          const int v = __float2int_rn(__fmul_rn(wxy, wzr));
          if constexpr (WIDE) atomicAdd(&acc[row + zz[rz]], (unsigned long long)(long long)v);
          else atomicAdd(&acc[row + zz[rz]], v);
        }
      }
    }
  }
}

// Two grids per pass share the entry loads and need no split of the packed
// spectra: deposit_fft_z 0.052 -> 0.034 ms (128^3, 1 M particles CIC), 0.135
// -> 0.127 (256^3, 1 M TSC); at 512^3 0.752 (4 Mi TSC, 4x4 instead of
// 8x4 tiles: 0.742 before, with twice the bucket fill), at 1024^3 6.87 -> 7.78
// (16 Mi PCS; the fill 1.28 -> 0.32).  Bound by the shared-memory pipe (0.71 of
// its wavefronts at 512^3), instruction issue (0.56 of the slots) and barriers.
//
// Deposit, z transform and row stores of one unit (steps 1-4 above); x0, y0:
// its first pencil.  WIDE: 64-bit cells.  sh[b]: bits given up by scale block
// b of the unit (its scale 2^(sg - sh[b]), sh[b] <= SH_MAX).  tm[grid]: the
// unit's exact totals at the common scale 2^sg (valid in thread 0).  SPILLED:
// the tile's spilled entries too.
template <int N, int MAS, int G, class CT, bool WIDE, bool SPILLED>
__device__ __forceinline__ void tile_unit(const DepGeom& g, const ColEntries& te, int sg,
                                          const int (&sh)[Unit<N, G, CT, WIDE>::NSB], int x0, int y0, int kz_cols,
                                          const float2* __restrict__ tw, float2* __restrict__ spec, unsigned char* smem,
                                          const unsigned* list, long long (*s_part)[G], long long (&tm)[G],
                                          bool clear) {
  using Cell = UnitCell<N, G, CT, WIDE>;
  using U = Unit<N, G, CT, WIDE>;
  constexpr int UY = U::UY, PAIRS = U::PAIRS, NT = U::NT, NSB = U::NSB;
  constexpr int P = N / 2 + 8, NX = G == 2 ? N : N / 2;
  constexpr int SBY = U::SBY;                                  // scale blocks along y
  Cell* acc = reinterpret_cast<Cell*>(smem);                   // [2 PAIRS][N] fixed-point cells
  float4* cs4 = reinterpret_cast<float4*>(smem);               // [PAIRS/2][N] slots of two columns, alias the cells
  const int tid = threadIdx.x;
  // 2^s of each block, and 2^-s times the packed transform's scale: s = sg - sh in [-110, 100], normal floats
  float up[NSB], dn[NSB];
#pragma unroll
  for (int b = 0; b < NSB; ++b) {
    up[b] = ldexpf(1.0f, sg - sh[b]);
    dn[b] = ldexpf(fft::PACK_SCALE<G>, sh[b] - sg);
  }

  if (clear) {
    uint4* a4 = reinterpret_cast<uint4*>(acc);
    for (int k = tid; k < (int)(U::CELLS * sizeof(Cell) / 16); k += NT) a4[k] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
  }
  // the entries whose places are kept, then the others (a loop that asks for each entry which it is: 512^3
  // deposit/z 750 -> 740 us)
#pragma unroll 1
  for (unsigned q = 0; q < 2; ++q) {
    const unsigned en = q ? te.n[0] : min(te.n[0], (unsigned)U::LIST);
    for (unsigned i = q * U::LIST + tid; i < en; i += NT)
      add_entry<N, MAS, G, CT, WIDE>(g, __ldg(te.entries + (q ? column_index(te, i) : list[i])), up, x0, y0, acc);
  }
  if constexpr (SPILLED)
    for_spilled<NT>(te.ctr->cat, te.n[1], [&](unsigned i) { return spilled_column(te, i); },
                    [&](const float4& e) { add_entry<N, MAS, G, CT, WIDE>(g, e, up, x0, y0, acc); });
  __syncthreads();

  // z transform: a thread transforms columns 2cp and 2cp+1 (one scale block), the same column pair in
  // every stage of the first (and only) butterfly per thread: cp = tid / (N/8).  The cells of column q:
  // the real parts at 2q N, the imaginary parts at (2q + 1) N
  auto block_of = [](int cp) {
    const int a = 2 * cp / UY, ly = 2 * cp % UY;
    return NSB == 1 ? 0 : ((G == 2 ? a : 2 * a) >> 2) * SBY + (ly >> 2);
  };
  long long part[G];
#pragma unroll
  for (int q = 0; q < G; ++q) part[q] = 0;
  auto gin = [&part, &dn, &sh, acc, block_of](int j, int cp) {
    const float d = pick_block<NSB>(block_of(cp), dn);
    const int f = 1 << pick_block<NSB>(block_of(cp), sh);     // the block's total at the common scale
    float v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const auto q = acc[(4 * cp + k) * N + j];
      // 32-bit cells: one widening multiply-add each
      part[G == 2 ? (k & 1) : 0] += (long long)q * f;
      v[k] = __fmul_rn(WIDE ? __ll2float_rn((long long)q) : __int2float_rn((int)q), d);   // exact: a power of two
    }
    return make_float4(v[0], v[1], v[2], v[3]);
  };
  auto sin_ = [cs4](int j, int cp) { return cs4[cp * N + fft::zsw(j)]; };
  auto sout = [cs4](int j, int cp, float4 v) { cs4[cp * N + fft::zsw(j)] = v; };
  // columns 2cp and 2cp + 1 are rows y0 + ly and y0 + ly + 1 of plane x0 + a (G = 2) or x0 / 2 + a
  auto gout = [spec, x0, y0, kz_cols](int k, int cp, float4 v) {
    const int a = 2 * cp / UY, ly = 2 * cp % UY;
    float2* o0 = spec + fft::PackedRows<N>::at((G == 2 ? x0 : x0 / 2) + a, y0 + ly);
    fft::store_packed<N>(o0, o0 + (long long)NX * N * P, fft::PackedRows<N>::ROW, kz_cols, k, v);
  };
  // 32-bit cells: the N / 8 threads of a column pair own its data (the first stage's writes alias the
  // pair's own pencils), so the stages synchronise groups of them only, a warp's or a named barrier
  // each.  64-bit cells span twice the bytes of the complex slots: whole-CTA barriers.
  constexpr int GS = WIDE ? 0 : fft::Z_GROUP<N>;
  static_assert(PAIRS * N / 16 <= NT, "one first-stage butterfly per thread");
  fft::run_stages2<N, PAIRS / 2, NT, true, true, false, decltype(gin), decltype(sin_), decltype(sout), decltype(gout),
                   GS>(gin, sin_, sout, gout, tw, tid);
  // the unit's exact totals
#pragma unroll
  for (int q = 0; q < G; ++q) {
    part[q] = warp_sum(part[q]);
    if ((tid & 31) == 0) s_part[tid >> 5][q] = part[q];
  }
  __syncthreads();                                     // also: the next unit reuses the accumulators
  if (tid < 32) {                                      // one warp: the block ends with this
#pragma unroll
    for (int q = 0; q < G; ++q) tm[q] = warp_sum(tid < NT / 32 ? s_part[tid][q] : 0ll);
  }
}

// Every unit of a tile; writes the tile's totals.  sh: the shifts of the tile's scale blocks.
template <int N, int MAS, int G, class CT, bool WIDE, bool SPILLED>
__device__ __forceinline__ void tile_units(const DepGeom& g, const ColEntries& te, int sg, const int (&sh)[CT::NSB],
                                           int x0, int y0, int kz_cols, const float2* __restrict__ tw,
                                           float2* __restrict__ spec, unsigned char* smem, const unsigned* list,
                                           long long (*s_part)[G], long long* tile_mass) {
  using U = Unit<N, G, CT, WIDE>;
  long long total[G];
#pragma unroll
  for (int q = 0; q < G; ++q) total[q] = 0;
#pragma unroll 1
  for (int u = 0; u < U::NU; ++u) {
    const int ux = u / U::NUY * U::UX, uy = u % U::NUY * U::UY;
    int shu[U::NSB];
    if constexpr (U::NU > 1) {
      static_assert(U::NU == 1 || U::NSB == 1, "a part of a tile lies in one scale block");
      shu[0] = pick_block<CT::NSB>((ux >> 2) * CT::SBY + (uy >> 2), sh);
    } else {
#pragma unroll
      for (int b = 0; b < U::NSB; ++b) shu[b] = sh[b];
    }
    long long tm[G];
    tile_unit<N, MAS, G, CT, WIDE, SPILLED>(g, te, sg, shu, x0 + ux, y0 + uy, kz_cols, tw, spec, smem, list,
                                                  s_part, tm, (WIDE && U::WIDE_WHOLE) || u > 0);
    if (threadIdx.x == 0) {
#pragma unroll
      for (int q = 0; q < G; ++q) total[q] += tm[q];
    }
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < G; ++q) tile_mass[(size_t)q * gridDim.x + blockIdx.x] = total[q];
  }
}

// The same with 64-bit cells, out of line: tiles of dense clumps are rare,
// and inlined their code would cost the others registers.  packed: 8 bits of
// shift per scale block.
template <int N, int MAS, int G, class CT>
__device__ __noinline__ void tile_units_wide(const DepGeom& g, ColEntries te, int sg, unsigned packed, int x0, int y0,
                                             int kz_cols, const float2* __restrict__ tw, float2* __restrict__ spec,
                                             long long (*s_part)[G], long long* tile_mass) {
  using U = Unit<N, G, CT, false>;
  extern __shared__ __align__(16) int acc_smem[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(acc_smem);
  const unsigned* list = reinterpret_cast<const unsigned*>(acc_smem + U::ROOM + CT::NSB * N);
  int sh[CT::NSB];
#pragma unroll
  for (int b = 0; b < CT::NSB; ++b) sh[b] = (int)((packed >> (8 * b)) & 0xffu);
  tile_units<N, MAS, G, CT, true, true>(g, te, sg, sh, x0, y0, kz_cols, tw, spec, smem, list, s_part, tile_mass);
}

// Adds entry e to the per-block plane counts zc [NSB][N] of the tile at
// (x0, y0).
template <int N, int MAS, int G, class CT>
__device__ __forceinline__ void count_planes(const DepGeom& g, const float4& e, int x0, int y0, int* zc) {
  constexpr int R = MAS, W = R + G - 1;
  // the union of the grids' nodes along each axis: first .. last (the second grid's first node
  // is the first grid's or the next one), as the bucketing counts them.  Every entry of the
  // bucket reaches the tile, so an axis with one block row needs no test
  int first[3], last[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    if ((a == 0 && CT::SBX == 1) || (a == 1 && CT::SBY == 1)) {
      first[a] = last[a] = 0;
      continue;
    }
    Axis<R> a0;
    make_axis<MAS, 0, N>(g, a == 0 ? e.x : (a == 1 ? e.y : e.z), 0, a0);
    first[a] = a0.first;
    last[a] = a0.first + R - 1;
    if constexpr (G == 2) {
      Axis<R> a1;
      make_axis<MAS, 0, N>(g, a == 0 ? e.x : (a == 1 ? e.y : e.z), 1, a1);
      last[a] = a1.first + R - 1;
    }
  }
  // scale blocks reached along x and y
  unsigned mx = CT::SBX == 1 ? 1u : 0u, my = CT::SBY == 1 ? 1u : 0u;
#pragma unroll
  for (int r = 0; r < W; ++r) {
    if constexpr (CT::SBX > 1) {
      const int cx = wrapn(first[0] + r, N) - x0;
      if (first[0] + r <= last[0] && cx >= 0 && cx < CT::TX) mx |= 1u << (cx >> 2);
    }
    if constexpr (CT::SBY > 1) {
      const int cy = wrapn(first[1] + r, N) - y0;
      if (first[1] + r <= last[1] && cy >= 0 && cy < CT::TY) my |= 1u << (cy >> 2);
    }
  }
#pragma unroll
  for (int bx = 0; bx < CT::SBX; ++bx)
#pragma unroll
    for (int by = 0; by < CT::SBY; ++by)
      if (((mx >> bx) & 1u) && ((my >> by) & 1u))
        for (int zn = first[2]; zn <= last[2]; ++zn) atomicAdd(&zc[(bx * CT::SBY + by) * N + wrapn(zn, N)], 1);
}

// Per-block plane counts of a tile (zc [NSB][N], zeroed on entry) and the
// bits each block gives up; returns true when some block is a dense clump
// (then sh[] holds SH_MAX + 1 for those blocks).  An entry covers block b in
// plane z when its nodes (any grid) reach b's 4 x-columns, its 4 y-columns
// and z.
template <int N, int MAS, int G, class CT, bool SPILLED>
__device__ __forceinline__ bool block_scales(const DepGeom& g, const ColEntries& te, int x0, int y0, int* zc,
                                             unsigned* list, int* s_max, int (&sh)[CT::NSB]) {
  constexpr int NT = Unit<N, G, CT, false>::NT, NSB = CT::NSB;
  constexpr unsigned LIST = Unit<N, G, CT, false>::LIST;
  const int tid = threadIdx.x;
  // this pass is the tile's first touch of its bucket: a thread issues EB entry loads at once
  constexpr int EB = 4;
#pragma unroll 1
  for (unsigned q = 0; q < 2; ++q) {                   // the entries whose places are kept, then the others
    const unsigned en = q ? te.n[0] : min(te.n[0], LIST);
    for (unsigned i0 = q * LIST + tid; i0 < en; i0 += EB * NT) {
      float4 ev[EB];
#pragma unroll
      for (int k = 0; k < EB; ++k) {
        const unsigned i = i0 + k * NT;
        ev[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < en) {
          const unsigned at = column_index(te, i);
          if (q == 0) list[i] = at;                    // read by this thread only, in the deposit
          ev[k] = __ldg(te.entries + at);
        }
      }
#pragma unroll
      for (int k = 0; k < EB; ++k) {
        if (i0 + k * NT >= en) break;
        count_planes<N, MAS, G, CT>(g, ev[k], x0, y0, zc);
      }
    }
  }
  if constexpr (SPILLED)
    for_spilled<NT>(te.ctr->cat, te.n[1], [&](unsigned i) { return spilled_column(te, i); },
                    [&](const float4& e) { count_planes<N, MAS, G, CT>(g, e, x0, y0, zc); });
  __syncthreads();
  // a node weight of TSC (<= 0.75^3) or PCS (<= (2/3)^3) is below 1/2: one more bit
  constexpr int WBIT = (MAS == GBP_TSC || MAS == GBP_PCS) ? 1 : 0;
  bool heavy = false;
#pragma unroll
  for (int b = 0; b < NSB; ++b) {
    int cmax = 0;
    for (int k = tid; k < N; k += NT) cmax = max(cmax, zc[b * N + k]);
    cmax = __reduce_max_sync(0xffffffffu, cmax);
    if ((tid & 31) == 0) s_max[tid >> 5] = cmax;
    __syncthreads();
    cmax = __reduce_max_sync(0xffffffffu, (tid & 31) < NT / 32 ? s_max[tid & 31] : 0);
    if (b + 1 < NSB) __syncthreads();                  // s_max is reused by the next block
    const unsigned cnt = (unsigned)cmax;
    const int lg = cnt > 1u ? 32 - __clz(cnt - 1u) : 0;  // ceil(log2(entries per plane))
    sh[b] = lg > WBIT ? lg - WBIT : 0;                 // block scale 2^(sg - sh), never finer than 2^sg
    if (sh[b] > SH_MAX) heavy = true;
  }
  return heavy;
}

// A tile's plane counts, scales and units; the cells and the plane counts are
// zero on entry.
template <int N, int MAS, int G, class CT, bool SPILLED>
__device__ __forceinline__ void column_tile(const DepGeom& g, const ColEntries& te, int sg, int x0, int y0, int kz_cols,
                                            const float2* __restrict__ tw, float2* __restrict__ spec,
                                            long long* __restrict__ tile_mass) {
  using U = Unit<N, G, CT, false>;
  constexpr int NT = U::NT, NSB = CT::NSB;
  extern __shared__ __align__(16) int acc_smem[];
  int* zc = acc_smem + U::ROOM;                       // [NSB][N] entries covering each block's planes
  unsigned* list = reinterpret_cast<unsigned*>(zc + NSB * N);
  __shared__ long long s_part[NT / 32][G];
  __shared__ int s_max[NT / 32];
  int sh[NSB];
  const bool heavy = block_scales<N, MAS, G, CT, SPILLED>(g, te, x0, y0, zc, list, s_max, sh);
  if (heavy) {                                         // uniform over the CTA
    unsigned packed = 0;
#pragma unroll
    for (int b = 0; b < NSB; ++b) packed |= (unsigned)(sh[b] > SH_MAX ? 0 : sh[b]) << (8 * b);
    tile_units_wide<N, MAS, G, CT>(g, te, sg, packed, x0, y0, kz_cols, tw, spec, s_part, tile_mass);
  } else {
    tile_units<N, MAS, G, CT, false, SPILLED>(g, te, sg, sh, x0, y0, kz_cols, tw, spec,
                                              reinterpret_cast<unsigned char*>(acc_smem), list, s_part, tile_mass);
  }
}

// A tile with spilled entries.
template <int N, int MAS, int G, class CT>
__device__ __noinline__ void column_spilled_tile(const DepGeom& g, ColEntries te, int sg, int x0, int y0, int kz_cols,
                                                 const float2* __restrict__ tw, float2* __restrict__ spec,
                                                 long long* __restrict__ tile_mass) {
  column_tile<N, MAS, G, CT, true>(g, te, sg, x0, y0, kz_cols, tw, spec, tile_mass);
}

template <int N, int MAS, int G, class CT>
__global__ void __launch_bounds__(Unit<N, G, CT, false>::NT, Unit<N, G, CT, false>::MINB)
deposit_fftz_kernel(const __grid_constant__ DepGeom g, const float4* __restrict__ entries,
                    const unsigned* __restrict__ counts, const __grid_constant__ Spill sp, DepCounters* ctr,
                    int kz_cols, const float2* __restrict__ tw, float2* __restrict__ spec,
                    long long* __restrict__ tile_mass) {
  pdl_wait();
  using U = Unit<N, G, CT, false>;
  constexpr int NT = U::NT;
  extern __shared__ __align__(16) int acc_smem[];
  __shared__ ColRuns s_runs;
  const int tid = threadIdx.x, t = blockIdx.x;
  const int ty = t % g.nt[1], tx = t / g.nt[1];
  const int x0 = tx * CT::TX, y0 = ty * CT::TY;
  for (int k = tid; k < (int)(U::CELLS / 4); k += NT)
    reinterpret_cast<uint4*>(acc_smem)[k] = make_uint4(0u, 0u, 0u, 0u);
  const ColEntries te = column_entries(g, tx, ty, entries, counts, sp, ctr, s_runs);
  if (tid == 0 && te.n[0] + te.n[1] > g.flag_cap) atomicOr(&ctr->outgrown, 1u);
  const int sg = fixed_scale_exp(ctr->maxw_bits, 0);
  for (int k = tid; k < CT::NSB * N; k += NT) acc_smem[U::ROOM + k] = 0;
  __syncthreads();
  if (te.n[1]) column_spilled_tile<N, MAS, G, CT>(g, te, sg, x0, y0, kz_cols, tw, spec, tile_mass);
  else column_tile<N, MAS, G, CT, false>(g, te, sg, x0, y0, kz_cols, tw, spec, tile_mass);
}

struct PartLayout {
  DepLayout dep;
  size_t xbin, total;
};

int particles_layout(int64_t n, gbp_fft_plan plan, gbp_bins B, int mas, int ells, int tx, int ty, PartLayout& L) {
  if (!plan || !B || plan->n != B->N) return GBP_ERR_INVALID;
  if (!plan->own || (plan->grids != 1 && plan->grids != 2)) return GBP_ERR_UNSUPPORTED;
  int st = column_layout(n, B->N, mas, plan->grids == 2, tx, ty, L.dep);
  if (st) return st;
  st = xbin_power_workspace(plan, B, ells, &L.xbin);
  if (st) return st;
  L.total = align256(L.dep.total) + L.xbin;
  return GBP_OK;
}

template <int N, int MAS, int G, class CT>
int run_fused(const DepGeom& g, const DepLayout& L, const DepBuffers& b, int kz_cols, const float2* tw, float2* spec,
              cudaStream_t st) {
  using U = Unit<N, G, CT, false>;
  int r = bucket_columns<MAS, G>(g, L, b, st);
  if (r) return r;
  auto k = deposit_fftz_kernel<N, MAS, G, CT>;
  GBP_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)U::SMEM));
  {
    GBP_TRACE("deposit_fft_z", st);
    GBP_CUDA_TRY(launch_pdl(k, dim3(L.ntiles), dim3(U::NT), U::SMEM, st, g, b.entries, b.counts, b.spill,
                            b.ctr, kz_cols, tw, spec, b.tile_mass));
  }
  return GBP_OK;
}

template <int N, class CT>
int dispatch_mas(int mas, int G, const DepGeom& g, const DepLayout& L, const DepBuffers& b, int kz_cols,
                 const float2* tw, float2* spec, cudaStream_t st) {
  if (G == 2) {
    switch (mas) {
      case GBP_NGP: return run_fused<N, GBP_NGP, 2, CT>(g, L, b, kz_cols, tw, spec, st);
      case GBP_CIC: return run_fused<N, GBP_CIC, 2, CT>(g, L, b, kz_cols, tw, spec, st);
      case GBP_TSC: return run_fused<N, GBP_TSC, 2, CT>(g, L, b, kz_cols, tw, spec, st);
      default: return run_fused<N, GBP_PCS, 2, CT>(g, L, b, kz_cols, tw, spec, st);
    }
  }
  switch (mas) {
    case GBP_NGP: return run_fused<N, GBP_NGP, 1, CT>(g, L, b, kz_cols, tw, spec, st);
    case GBP_CIC: return run_fused<N, GBP_CIC, 1, CT>(g, L, b, kz_cols, tw, spec, st);
    case GBP_TSC: return run_fused<N, GBP_TSC, 1, CT>(g, L, b, kz_cols, tw, spec, st);
    default: return run_fused<N, GBP_PCS, 1, CT>(g, L, b, kz_cols, tw, spec, st);
  }
}

// The whole fused path for mesh side N: bucketing, deposit + z pass, y pass,
// x pass + binning.  (tx, ty) is a supported tile shape for N (checked by
// the caller).
template <int N>
int particles_power_n(DepGeom g, int64_t n_launch, gbp_fft_plan plan, gbp_bins B, int mas, int ells, int tx, int ty,
                      void* spectrum, double* sums_out, long long* nmodes_out, double* ksum_out,
                      gbp_deposit_stats* stats_out, void* workspace, size_t ws_bytes, cudaStream_t st) {
  if (!spectrum || !sums_out || !nmodes_out || !stats_out) return GBP_ERR_INVALID;
  if ((reinterpret_cast<uintptr_t>(spectrum) & 15u) != 0) return GBP_ERR_INVALID;
  PartLayout L;
  int r = particles_layout(n_launch, plan, B, mas, ells, tx, ty, L);
  if (r) return r;
  if (!workspace || ws_bytes < L.total) return GBP_ERR_WORKSPACE;
  const DepBuffers b = carve_deposit(workspace, L.dep);
  void* xws = static_cast<char*>(workspace) + align256(L.dep.total);
  for (int a = 0; a < 3; ++a) { g.td[a] = L.dep.td[a]; g.ts[a] = L.dep.ts[a]; g.nt[a] = L.dep.nt[a]; }
  g.vec_ok = 0;
  g.tcap = L.dep.tcap;
  g.flag_cap = L.dep.flag_cap;
  for (int c = 0; c < 4; ++c) { g.ccap[c] = L.dep.ccap[c]; g.coff[c] = L.dep.coff[c]; }
  const int G = plan->grids;
  float2* spec = static_cast<float2*>(spectrum);
  GBP_CUDA_TRY(cudaMemsetAsync(b.ctr, 0, zeroed_bytes(L.dep), st));
  r = GBP_ERR_UNSUPPORTED;
  if (tx == 4 && ty == 4) {
    r = dispatch_mas<N, ColTile<N, 4, 4>>(mas, G, g, L.dep, b, B->kz_cols, plan->tw, spec, st);
  } else if (tx == 8 && ty == 4) {
    if constexpr (N <= 512) r = dispatch_mas<N, ColTile<N, 8, 4>>(mas, G, g, L.dep, b, B->kz_cols, plan->tw, spec, st);
  } else if (tx == 8 && ty == 8) {
    if constexpr (N == 128 || N == 256)
      r = dispatch_mas<N, ColTile<N, 8, 8>>(mas, G, g, L.dep, b, B->kz_cols, plan->tw, spec, st);
  }
  if (r) return r;
  // up to 256^3 the statistics are a block of the last fold (as fast as a kernel of its own less the launch,
  // 3 us at 256^3, 2 % of a 128^3 batch); beyond, that block would outlast the fold (1024^3: 78 against 29 + 20 us)
  StatsFold stats = stats_fold(b, L.dep, GBP_COMPAT_NONE, G, stats_out);
  if (N > 256) {
    r = deposit_stats(b, L.dep, GBP_COMPAT_NONE, G, stats_out, st);
    if (r) return r;
    stats.out = nullptr;
  }
  r = own_fft_y_packed(N, G, spec, B->kz_cols, B->last_closed, plan->tw, st);
  if (r) return r;
  const double* mass = reinterpret_cast<const double*>(stats_out);   // gbp_deposit_stats starts with mass[2]
  return xbin_power(plan, spec, B, mas, ells, mass, sums_out, nmodes_out, ksum_out, xws, L.xbin, st, stats);
}

}  // namespace
}  // namespace gbp

// One translation unit per mesh side defines these (no reference
// counterpart; depfft.cu's C ABI calls them).  The job pointer, when
// non-null, replaces x, y, z, w, n and the box geometry (capacity = n).
#define GBP_DEPFFT_INSTANCE(NN)                                                                                    \
  namespace gbp {                                                                                                  \
  int particles_ws_n##NN(int64_t n, gbp_fft_plan plan, gbp_bins bins, int mas, int ells, int tx, int ty,           \
                         size_t* bytes) {                                                                          \
    PartLayout L;                                                                                                  \
    const int st = particles_layout(n, plan, bins, mas, ells, tx, ty, L);                                          \
    if (st) return st;                                                                                             \
    *bytes = L.total;                                                                                              \
    return GBP_OK;                                                                                                 \
  }                                                                                                                \
  int particles_power_n##NN(const float* x, const float* y, const float* z, const float* w, int64_t n, float xmin, \
                            float ymin, float zmin, float inv_cell, const gbp_job* job, gbp_fft_plan plan,        \
                            gbp_bins bins, int mas, int ells, int tx, int ty, void* spectrum, double* sums_out,    \
                            long long* nmodes_out, double* ksum_out, gbp_deposit_stats* stats_out,                 \
                            void* workspace, size_t ws_bytes, cudaStream_t st) {                                   \
    DepGeom g{};                                                                                                   \
    g.x = x; g.y = y; g.z = z; g.w = w; g.n = n;                                                                   \
    g.ox = xmin; g.oy = ymin; g.oz = zmin; g.inv_cell = inv_cell;                                                  \
    g.N = NN;                                                                                                      \
    g.job = job;                                                                                                   \
    g.cap = n;                                                                                                     \
    return particles_power_n<NN>(g, n, plan, bins, mas, ells, tx, ty, spectrum, sums_out, nmodes_out, ksum_out,   \
                                 stats_out, workspace, ws_bytes, st);                                              \
  }                                                                                                                \
  }
