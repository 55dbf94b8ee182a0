// Column-FFT engine shared by every pass of the library transform: radix-8
// Stockham stages (fft_core.cuh) over blocks of columns, where
//
//   * each thread transforms the same butterfly of two adjacent columns at
//     once: every shared or global access moves 16 bytes (two complex
//     values), the two butterflies share one set of twiddle factors, and
//     their additions are single f32x2 instructions (values that cross shared
//     memory between stages are kept as two real and two imaginary parts, so
//     they need no rearranging): 1-4 % of each pass;
//   * the twiddles come from per-stage tables, w_r(k) = exp(-2 pi i r k /
//     (R p)) for r < 8 stored contiguously per k (four 16-byte loads);
//   * the first stage reads its inputs from wherever they are (HBM, or
//     integer accumulators) and the last stage writes its outputs to
//     wherever they go (HBM, or a transposed shared buffer); only the
//     exchanges between stages go through shared memory.
//
// Two shared layouts, both free of bank conflicts for every stage's access
// pattern (checked by enumeration):
//
//   ColBlock (thread b owns column pair b % CP, butterfly b / CP): row j of a
//     block of 8 columns is 64 bytes, stored at physical row j ^ bit3(j), so
//     the two rows of a quarter-warp fall on the two halves of a 128-byte
//     bank line; two slabs (two grids) are offset by 64 bytes.
//   Column-major pairs (IFAST: consecutive lanes on consecutive rows): the
//     16-byte slot of rows j of two adjacent columns is at j ^ ((j >> 3) & 7),
//     so 8 consecutive rows of any stage (the stride-8 writes of the first
//     stage included) hit 8 distinct slots.
//
// Forward transform exp(-2 pi i j k / N) (cuFFT, numpy), natural-order output.
#pragma once

#include "fft_core.cuh"

namespace gbp {
namespace fft {

// Offset (in float2) of the twiddle table of the stage with span p > 1; the
// first N entries of the table buffer are exp(-2 pi i e / N).
template <int N>
__host__ __device__ constexpr int tw_off(int p) { return N + 8 * (p - 8) / 7; }

// Size (in float2) of the whole twiddle buffer for N.
template <int N>
constexpr int tw_size() {
  int p = 1;
  for (int s = 0; s < Radices<N>::n8; ++s) p *= 8;   // span of the last radix-8 stage's successor
  return tw_off<N>(p) + 8 * p;
}

__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 pack2(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }

// Barrier of the GS consecutive threads that share data (a named barrier,
// id 1 + tid / GS), or of the whole CTA when GS == 0.
// A CTA has 16 named barriers and __syncthreads is number 0: at most 15 groups.
constexpr int MAX_GROUPS = 15;

// Threads of a group that owns whole column pairs (N / 8 threads each, at least a warp), and the rule of the z
// passes: from 512 up, where a pair's threads are two warps or more, groups (deposit and z pass at 1024^3, one CTA of
// 1024 threads per SM: 7.95 -> 7.78 ms); below, a CTA barrier keeps a block's loads and stores together (256^3, two
// meshes: z 0.053 ms, inverse 0.051; with a warp per pair 0.056 and 0.055).
template <int N>
constexpr int GROUP = N / 8 < 32 ? 32 : N / 8;
template <int N>
constexpr int Z_GROUP = N >= 512 ? GROUP<N> : 0;

template <int GS>
__device__ __forceinline__ void group_sync(int tid) {
  if constexpr (GS == 0) {
    __syncthreads();
  } else if constexpr (GS == 32) {
    __syncwarp();
  } else {
    static_assert(GS % 32 == 0, "named barriers count whole warps");
    asm volatile("bar.sync %0, %1;" ::"r"(1 + tid / GS), "n"(GS) : "memory");
  }
}

// One stage over CP column pairs.  In(row, cp) -> float4, Out(row, cp, float4).
// MID_SYNC separates the reads from the writes (in-place shared stages);
// END_SYNC publishes the writes.  IFAST: thread b owns butterfly b % (N/R) of
// column pair b / (N/R) (consecutive lanes, consecutive rows); otherwise
// column pair b % CP, butterfly b / CP.  GS > 0 (IFAST, N / 8 threads per
// column pair): a group of GS threads owns GS * 8 / N column pairs, whose data
// no other thread touches, and the barriers cover the group only.
// PLANAR_IN / PLANAR_OUT: a
// float4 holds (re, re, im, im) of the two columns, else (re, im, re, im).
template <int N, int R, int CP, int NT, bool MID_SYNC, bool END_SYNC, bool IFAST, bool PLANAR_IN, bool PLANAR_OUT,
          class In, class Out, int GS = 0>
__device__ __forceinline__ void stage2(In in, Out out, const float2* __restrict__ tw, int p, int tid) {
  constexpr int NB = CP * (N / R);
  constexpr int PER = GS > 0 ? 8 / R : (NB + NT - 1) / NT;
  static_assert(GS == 0 || (IFAST && GS == GROUP<N> && CP * (N / 8) % (GS > 0 ? GS : 1) == 0 && CP * (N / 8) <= NT),
                "whole groups, one first-stage butterfly per thread");
  static_assert(GS <= 32 || NT / (GS > 0 ? GS : 1) <= MAX_GROUPS, "more groups than named barriers");
  // number of butterfly q of the thread, column pair by column pair
  constexpr int STEP = GS > 0 ? GS : NT;
  const int b0 = GS > 0 && PER > 1 ? tid + tid / STEP * STEP * (PER - 1) : tid;
  auto number = [b0](int q) { return b0 + q * STEP; };
  float4 u[PER][R];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int b = number(q);
    if (PER * NT != NB && b >= NB) continue;
    const int cp = IFAST ? b / (N / R) : b % CP, i = IFAST ? b % (N / R) : b / CP;
#pragma unroll
    for (int r = 0; r < R; ++r) u[q][r] = in(i + r * (N / R), cp);
    Pair a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float4 v = u[q][r];
      a[r] = PLANAR_IN ? Pair{make_float2(v.x, v.y), make_float2(v.z, v.w)}
                       : Pair{make_float2(v.x, v.z), make_float2(v.y, v.w)};
    }
    if (p > 1) {
      const int k = i & (p - 1);
      const float4* t4 = reinterpret_cast<const float4*>(tw + tw_off<N>(p) + k * 8);
#pragma unroll
      for (int rr = 0; rr < R / 2; ++rr) {
        const float4 w = __ldg(t4 + rr);
        if (rr > 0) a[2 * rr] = cmul(a[2 * rr], lo2(w));
        a[2 * rr + 1] = cmul(a[2 * rr + 1], hi2(w));
      }
    }
    if constexpr (R == 8) dft8(a);
    else if constexpr (R == 4) dft4(a);
    else dft2(a[0], a[1]);
#pragma unroll
    for (int r = 0; r < R; ++r)
      u[q][r] = PLANAR_OUT ? make_float4(a[r].re.x, a[r].re.y, a[r].im.x, a[r].im.y)
                           : make_float4(a[r].re.x, a[r].im.x, a[r].re.y, a[r].im.y);
  }
  if (MID_SYNC) group_sync<GS>(tid);
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int b = number(q);
    if (PER * NT != NB && b >= NB) continue;
    const int cp = IFAST ? b / (N / R) : b % CP, i = IFAST ? b % (N / R) : b / CP;
    const int k = i & (p - 1);
    const int j = (i - k) * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) out(j + r * p, cp, u[q][r]);
  }
  if (END_SYNC) group_sync<GS>(tid);
}

// Full transform: the first stage reads `gin`, the stages in between go
// through shared memory (`sin` / `sout`), the last stage writes `gout`.
// Starts without a barrier (the caller orders earlier uses of shared
// memory).  IN_SHARED: `gin` reads shared memory that the first stage's
// writes alias; OUT_SHARED: `gout` writes the shared memory the last stage
// reads (each then reads everything before it writes; OUT_SHARED also ends
// with a barrier).
template <int N, int CP, int NT, bool IFAST, bool IN_SHARED, bool OUT_SHARED, class GIn, class SIn, class SOut,
          class GOut, int GS = IFAST ? Z_GROUP<N> : 0>
__device__ __forceinline__ void run_stages2(GIn gin, SIn sin_, SOut sout, GOut gout, const float2* __restrict__ tw,
                                            int tid) {
  using RD = Radices<N>;
  static_assert(RD::stages >= 2, "at least two stages");
  stage2<N, 8, CP, NT, IN_SHARED, true, IFAST, false, true, GIn, SOut, GS>(gin, sout, tw, 1, tid);
  int p = 8;
  if constexpr (RD::tail == 0) {
#pragma unroll
    for (int st = 1; st < RD::n8 - 1; ++st) {
      stage2<N, 8, CP, NT, true, true, IFAST, true, true, SIn, SOut, GS>(sin_, sout, tw, p, tid);
      p *= 8;
    }
    // the last stage's outputs may be read by any thread: a CTA barrier ends it
    stage2<N, 8, CP, NT, OUT_SHARED, false, IFAST, true, false, SIn, GOut, GS>(sin_, gout, tw, p, tid);
    if (OUT_SHARED) __syncthreads();
  } else {
#pragma unroll
    for (int st = 1; st < RD::n8; ++st) {
      stage2<N, 8, CP, NT, true, true, IFAST, true, true, SIn, SOut, GS>(sin_, sout, tw, p, tid);
      p *= 8;
    }
    constexpr int R = RD::tail == 1 ? 2 : 4;
    stage2<N, R, CP, NT, OUT_SHARED, false, IFAST, true, false, SIn, GOut, GS>(sin_, gout, tw, p, tid);
    if (OUT_SHARED) __syncthreads();
  }
}

// Blocks of 8 columns (x SLABS); a float4 holds two adjacent columns.
template <int N, int SLABS>
struct ColBlock {
  static constexpr int COLS = 8 * SLABS;
  static constexpr int CP = COLS / 2;
  static constexpr int SLAB = N * 8 + 8;    // complex per slab (+8: the 64-byte shift of slab 1)
  __device__ static __forceinline__ int row(int j) { return SLABS == 1 ? (j ^ ((j >> 3) & 1)) : j; }
  // float4 index of column pair cp (columns 2cp, 2cp+1) in row j
  __device__ static __forceinline__ int at(int j, int cp) { return (cp >> 2) * (SLAB / 2) + row(j) * 4 + (cp & 3); }
};

// IN_SHARED: the first stage's shared-memory writes must wait for earlier
// readers of `s` (a barrier between its loads and its writes), so a caller
// can start the loads of the next block while other warps still read the
// previous one.
template <int N, int SLABS, int NT, bool OUT_SHARED, class In, class Out, bool IN_SHARED = false>
__device__ __forceinline__ void col_fft(float2* s, In gin, Out gout, const float2* __restrict__ tw, int tid) {
  using L = ColBlock<N, SLABS>;
  float4* s4 = reinterpret_cast<float4*>(s);
  auto sin_ = [s4](int j, int cp) { return s4[L::at(j, cp)]; };
  auto sout = [s4](int j, int cp, float4 v) { s4[L::at(j, cp)] = v; };
  run_stages2<N, L::CP, NT, false, IN_SHARED, OUT_SHARED>(gin, sin_, sout, gout, tw, tid);
}

// Rows of a packed spectrum (slabs of x planes, rows y, N/2 + 8 complex kz):
// W planes are interleaved in blocks of 8 kz (64 bytes), so the x pass, which
// reads one block of every plane, finds W of them side by side.  Its time at
// 512^3, two grids: W = 1 0.527 ms, 2 0.458, 4 0.438, all planes 0.435.  N and
// N / 2 planes of a slab are multiples of 4.
constexpr int PACK_W = 4;
template <int N, int W = PACK_W>
struct PackedRows {
  static constexpr int P = N / 2 + 8, ROW = W * P, BLOCK = 8 * W;      // from a row, a kz block, to the next
  __device__ static __forceinline__ long long plane(int x) {
    return (long long)(x / W) * W * N * P + (x % W) * 8;
  }
  __device__ static __forceinline__ long long at(int x, int y) { return plane(x) + (long long)y * ROW; }
  __device__ static __forceinline__ int kz(int k) { return (k >> 3) * BLOCK + (k & 7); }
};

// Scale of the fields that the z passes of the packed transform read: with it
// unpack_mode (xpass.cuh) gives the mode F(k), or (F0 + phi F1) / 2 of two
// grids, itself, and its square overflows no earlier than |F|^2 does (a power
// of two: the same bits as a factor on the square).
template <int G>
constexpr float PACK_SCALE = G == 2 ? 0.25f : 0.5f;

// Stores Z[k] of two columns of a packed z pass, whose entries lie `step`
// apart: kz = k goes to slab 0 (o0) when k <= N/2, kz = -(N - k) to slab 1
// (o1) as entry N - k when N - k <= N/2; only kz < kz_cols are kept.
template <int N>
__device__ __forceinline__ void store_packed(float2* o0, float2* o1, int step, int kz_cols, int k, float4 v) {
  using R = PackedRows<N>;
  const int m = (N - k) & (N - 1);
  if (k <= N / 2 && k < kz_cols) {
    __stcs(o0 + R::kz(k), lo2(v));
    __stcs(o0 + step + R::kz(k), hi2(v));
  }
  if (m <= N / 2 && m < kz_cols) {
    __stcs(o1 + R::kz(m), lo2(v));
    __stcs(o1 + step + R::kz(m), hi2(v));
  }
}

// Slot of row j in a column-major block of column pairs (IFAST stages).
__device__ __forceinline__ int zsw(int j) { return j ^ ((j >> 3) & 7); }

}  // namespace fft
}  // namespace gbp
