// window.cuh -- window extremes (min, max or both) and window sums along a line for any reach, sm_103a.
//
// Van Herk / Gil-Werman with blocks shorter than the window: a line is cut into blocks of B
// entries; a window [e - 2r, e] is the suffix of the block its first entry lies in, whole blocks,
// and the prefix up to e of the block e lies in.  The thread that holds a block keeps its entries
// (and so every prefix) in registers and stores the block's suffixes to a ring in shared memory; a
// window then costs one suffix load, and the whole blocks between come from their first suffixes
// once per block (at most two different runs of them).  With blocks as long as the window (2r + 1
// entries) few threads share a line's serial work and the registers bound the reach; with
// blocks of 8 or 16 every thread's chain is short and the reach only sets the ring's length.
//
// Every entry a window combines lies in the window, so no neutral element is needed; the two
// halves overlap freely, min and max do not round, and the order of combination does not matter.
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace hdog {

constexpr int kExtCols = 32;   // columns of a ext_cols block, one per lane

// Rows of ext_cols' ring: the window's reach back, and two chunks (one being read, one written).
__host__ __device__ constexpr int ext_cols_rows(int r, int B, int NW) { return (2 * r + B - 1) / B * B + 2 * NW * B; }

// Lines across the lanes (along y or z): threadIdx.x is the column, threadIdx.y one of NW warps, each of which
// takes B consecutive entries of the 32 columns at a time.  Entry u of a line (u = 0 .. n + 2r - 1)
// is the input at line position t0 - r + u; output t (t = 0 .. n - 1) is the extreme of entries
// t .. t + 2r.  load(a, v): entries a .. a + B - 1 into v (a < n + 2r; entries past the line's last are
// not used); store(t, m).  Needs 2r >= B.  ring: ext_cols_rows(r, B, NW) x 32 values.
template <class Op, int B, int NW, class LoadF, class StoreF>
__device__ __forceinline__ void ext_cols(typename Op::T *ring, int n, int r, LoadF load, StoreF store) {
  using T = typename Op::T;
  const int lane = threadIdx.x, w = threadIdx.y;
  const int rows = ext_cols_rows(r, B, NW), total = n + 2 * r;
  const int back = (2 * r + B - 1) / B;    // blocks from e's to the one a window starts in (the first B - q outputs)
  const int q = back * B - 2 * r;          // that window's place in its first block
  int pos = w * B;
  for (int c = 0; c < total; c += NW * B) {
    const int a = c + w * B;
    T v[B];
    if (a < total) {
      load(a, v);
      T s = v[B - 1];
      ring[(pos + B - 1) * 32 + lane] = s;
#pragma unroll
      for (int j = B - 2; j >= 0; j--) {
        s = Op::op(v[j], s);
        ring[(pos + j) * 32 + lane] = s;
      }
    }
    __syncthreads();   // one a chunk: the ring holds the chunk after this one beside what this one reads
    if (a < total && a + B > 2 * r) {
      auto blk = [&](int d) {
        int p = pos - d * B;
        p += p < 0 ? rows : 0;
        return ring + p * 32 + lane;
      };
      T mid1 = v[0];                        // entry a is in every window that ends in this block
      for (int d = back - 2; d >= 1; d--) mid1 = Op::op(mid1, *blk(d));
      T mid0 = mid1;
      if (back >= 2) mid0 = Op::op(mid0, *blk(back - 1));
      const T *s0 = blk(back) + q * 32, *s1 = back >= 2 ? blk(back - 1) + (q - B) * 32 : s0;
      T p = v[0];
#pragma unroll
      for (int o = 0; o < B; o++) {
        if (o) p = Op::op(p, v[o]);
        const int e = a + o;
        const bool first = o < B - q;
        if (e >= 2 * r && e < total) store(e - 2 * r, Op::op(Op::op(p, first ? mid0 : mid1), (first ? s0 : s1)[o * 32]));
      }
    }
    pos += NW * B;
    if (pos >= rows) pos -= rows;
  }
}

// Lines along x: a group of G lanes per line (32 / G lines per warp), the group's lane l taking the 8
// entries 8 l .. 8 l + 7 of each chunk of 8 G.  Entry 8 b + o of a line lies in the ring at
// [o][line of the warp][b % NB]: the lanes' own accesses, and those of a window start, which lies the
// same number of entries back for every lane, spread over the banks (NB = 24 for G = 8: four lines of
// 8 lanes start 8 banks apart).
template <int G>
struct RowRing {
  static constexpr int LINES = 32 / G, CHUNK = 8 * G;
  // blocks kept per line: whole chunks, at least one and a window's reach back (8 blocks for G = 8, 64 for 32)
  static constexpr int NB = G == 8 ? 24 : 96;
  static constexpr int PITCH = LINES * NB;            // words between o and o + 1
  static constexpr int WORDS = 8 * PITCH;
  static constexpr int MAX_R = G == 8 ? 31 : 255;     // window of 2r + 1 entries within the reach
};

// Whether 8 lanes a row serve a pass best, or 32.  Eight waste less of a short row's last chunk and start four rows a
// warp, but a row then takes four times as many steps one after the other, which only many rows hide: from 32 rows per SM
// on, 64 where rows are long.  us with 8 / 32 lanes at reach 20: min/max and box of 2560 columns 33/20 in 2160 rows,
// 71/60 in 9728; of 256 columns 12/10 in 2160, 14/18 in 8192, 62/109 in 69120.  narrow: rows wider than this never
// take 8 lanes (the erosion's chunks carry little: 128 columns 29/30 in 69120 rows, 256 columns 52/49).
inline bool row_of_8(int r, int W, int64_t rows, int narrow) {
  return r <= RowRing<8>::MAX_R && W <= narrow && rows >= (W <= 1024 ? 32 : 64) * 152;
}

// The value of the group's lane `lag` lanes back (1 .. G): cur in this chunk, prev in the one before.
template <int G, class T>
__device__ __forceinline__ T row_lag(T cur, T prev, int lag) {
  const int gl = threadIdx.x & (G - 1);
  return __shfl_sync(0xFFFFFFFFu, gl >= G - lag ? prev : cur, (gl - lag) & (G - 1), G);
}

template <int G>
__device__ __forceinline__ float2 row_lag(float2 cur, float2 prev, int lag) {
  return make_float2(row_lag<G>(cur.x, prev.x, lag), row_lag<G>(cur.y, prev.y, lag));
}

// A ring seen from the lane's block of the chunk that starts at block pc: at(d) is the block d blocks back.
template <int G>
struct RowAt {
  int pc, base;   // base: the line's first word
  __device__ __forceinline__ RowAt(int pc_) : pc(pc_), base(((threadIdx.x & 31) / G) * RowRing<G>::NB) {}
  __device__ __forceinline__ int operator()(int d) const {
    const int b = pc + (int)(threadIdx.x & (G - 1)) - d;
    return base + (b < 0 ? b + RowRing<G>::NB : b);
  }
};

// The window extremes of one chunk.  v: the lane's 8 entries; suf: the ring; pc: the chunk's first block in it;
// hist: per doubling step the previous chunk's values (kept by the caller).  m[o] becomes the extreme of
// the 2r + 1 entries that end with the lane's entry o.  4 <= r <= MAX_R; Q = 8 ceil(2r / 8) - 2r.
template <class Op, int G, int Q>
__device__ __forceinline__ void ext_row_chunk(typename Op::T *suf, int pc, int r, const typename Op::T (&v)[8],
                                              typename Op::T (&hist)[6], typename Op::T (&m)[8]) {
  using T = typename Op::T;
  using R = RowRing<G>;
  const RowAt<G> at(pc);
  const int own = at(0);
  T s = v[7];
  suf[7 * R::PITCH + own] = s;
#pragma unroll
  for (int o = 6; o >= 0; o--) {
    s = Op::op(v[o], s);
    suf[o * R::PITCH + own] = s;
  }
  const int back = (2 * r + 7) / 8;
  __syncwarp();
  // whole blocks 1 .. back - 2 behind the lane's: two runs of 2^k blocks from doubling (a run ending at the lane's
  // own block joins the one that ends 2^k blocks before)
  T mid1 = v[0], d = s;
  const int n1 = back - 2;
#pragma unroll
  for (int k = 0; k < (G == 8 ? 3 : 6); k++) {
    if ((1 << k) <= n1) {
      const bool last = (2 << k) > n1;
      if (last) mid1 = Op::op(mid1, Op::op(row_lag<G>(d, hist[k], 1), row_lag<G>(d, hist[k], 1 + n1 - (1 << k))));
      const T h = hist[k];
      hist[k] = d;
      if (!last) d = Op::op(d, row_lag<G>(d, h, 1 << k));
    }
  }
  T mid0 = mid1;
  if (back >= 2) mid0 = Op::op(mid0, suf[at(back - 1)]);
  const T *s0 = suf + at(back), *s1 = suf + at(back >= 2 ? back - 1 : 1);
  T p = v[0];
#pragma unroll
  for (int o = 0; o < 8; o++) {
    if (o) p = Op::op(p, v[o]);
    if (Q + o < 8) m[o] = Op::op(Op::op(p, mid0), s0[(Q + o) * R::PITCH]);
    else m[o] = Op::op(Op::op(p, mid1), s1[(Q + o - 8) * R::PITCH]);
  }
}

// a / n for an odd whole number n below 2^20, correctly rounded for every finite a (a window's length): with z = 1 / n
// rounded and q = a z rounded, q + r z rounds to the quotient, r = a - n q being the remainder (P. Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990).  q is within two units in
// its last place, u, of a / n, and a and n q are multiples of u (of 2^-149 among the subnormals), so r is one too, of at
// most 2n of them, and exact in one FMA.  a / n - q is then k u / n for a whole k, which for odd n stays at least u / (4n)
// away from every rounding midpoint, while r z differs from it by less than u / 2^22.  An infinite or NaN a leaves no
// remainder to correct with; a zero's sign is not kept (sums that start at +0 never are -0).
struct SoftDiv {
  float n, z;
  __device__ __forceinline__ SoftDiv(int n_) : n((float)n_), z(1.0f / (float)n_) {}
  __device__ __forceinline__ float2 operator()(float2 a) const {
    const float2 zz = make_float2(z, z), q = mul2(a, zz), r = fma2(make_float2(-n, -n), q, a), p = fma2(r, zz, q);
    return make_float2(r.x == r.x ? p.x : q.x, r.y == r.y ? p.y : q.y);
  }
};

// Register-blocked sequential sums: a thread produces K consecutive outputs along the
// axis; slot (u + k) % K of a K-entry rotating window feeds output k at tap u of each
// block of K taps, so the window never moves between registers.  Every output still
// sums its 2r+1 inputs from 0.0f in the reference order.  load(i) returns input
// c0 - r + i, i = 0 .. L + K - 2 in order: an even K never divides the odd L, so the last block of
// taps is the guarded one and no load goes past the last window.
template <int K, class LoadF>
__device__ __forceinline__ void box_chain(int L, LoadF load, float2 (&acc)[K]) {
  static_assert(K % 2 == 0, "an odd K could divide L and load one input past the last window");
  float2 win[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    win[k] = load(k);
    acc[k] = make_float2(0.f, 0.f);
  }
  int jb = 0;
  for (; jb + K <= L; jb += K) {
#pragma unroll
    for (int u = 0; u < K; u++) {
#pragma unroll
      for (int k = 0; k < K; k++) acc[k] = add2(acc[k], win[(u + k) % K]);
      win[u] = load(jb + u + K);
    }
  }
#pragma unroll
  for (int u = 0; u < K; u++) {
    if (jb + u < L) {
#pragma unroll
      for (int k = 0; k < K; k++) acc[k] = add2(acc[k], win[(u + k) % K]);
      if (jb + u + K < L + K - 1) win[u] = load(jb + u + K);
    }
  }
}

}  // namespace hdog
