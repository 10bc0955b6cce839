// sweep.cu -- DoG and Hessian + negative-definite test as two z-sweeps over xy tiles, sm_103a.
//
// Reference: src/3D/DoG3DFilter.cu (DoG3DFilter :431-437: x -> y -> z separable Gaussians
// with zero borders, `(small - large) * normalizer`) and src/3D/Hessian3DFilter_element.cu
// (HessianPositiveDefiniteWithElement :355-388: gradients of gradients with zero halos,
// Sylvester test).  The reference runs 16 full-volume passes here and keeps the DoG and
// six Hessian planes in memory; the sweeps write the DoG volume, the uint8 mask and a compact
// list of the foreground voxels' Hessian elements.  The DoG sweep is specialised on the tap radii;
// other radii take the separate passes of dog.cu, and the Hessian sweep serves both.
// Every wait on a TMA barrier is bounded; a timeout sets HDOG_ERR_TIMEOUT and the
// kernel finishes without further waits.
#include <cuda.h>

#include <algorithm>

#include <type_traits>

#include "kernels.cuh"

namespace hdog {

// One normalized slice (box bw x bh at (x, y, z, s)) into shared memory.
__device__ __forceinline__ void tma_slice(const CUtensorMap *map, float *dst, uint64_t *bar, int x, int y, int z, int s,
                                          uint32_t bytes) {
  tma_load_4d(map, dst, bar, x, y, z, s, bytes);
}

// ------------------------------------------------------------------ radius-specialised sweeps
// For common sigma pairs the chain runs as two z-sweeps with the four tap radii as
// template parameters (RA/RB: xy radius of the small/large scale, ZA/ZB: z radius):
//
//   k_dog_sweep   normalized -> DoG volume.  A block owns a 32 x 24 tile (32 x 16 of
//                 a small batch) and sweeps
//                 z; stage A filters slice it along x (TMA-loaded, double-buffered), stage
//                 B filters slice it-1 along y and feeds the z shift register, which emits
//                 DoG slice it-1-RZ straight to global memory.  One barrier per slice.
//                 Tap pairs shared by both scales sit in per-thread registers, the taps of
//                 the wider scale alone are constant-bank operands.  The z shift
//                 register never moves: output zo lives in slot zo mod (2RZ+1), and the loop
//                 is unrolled over one turn, so the slot of every tap is known when compiling.
//                 Every output is the reference's FMA chain, zero taps at the borders
//                 included, so the volume equals the separate passes bit for bit.
//   k_hess_sweep  DoG -> mask + foreground list.  A block owns a kHTX x kHTY tile; DoG slices
//                 (tile + 2-voxel halo, zero outside the volume) arrive by TMA into an
//                 ring of six or eight slots, as far ahead; each thread tests an x quad of one or two rows.  No
//                 block barrier per slice: warps release ring slots through mbarriers.
//                 The normalized values the list carries are read from global memory by
//                 the threads whose quad has foreground.
//
// The split costs one write and one read of the DoG volume but frees the Hessian stage
// from the z shift register's registers, so several Hessian blocks share an SM.
constexpr int kDTX = 32;                // DoG tile width
constexpr int kHTX = 32, kHTY = 16;     // Hessian tile
constexpr int kHPX = kHTX + 8;          // Hessian ring row: columns x0-4 .. x0+kHTX+3 (16-byte aligned start)
constexpr int kHPY = kHTY + 4;
// Staged list entries per warp: one iteration adds at most 128 (four voxels per lane).
constexpr int kHStage = 128;
// Rows of an x quad that a thread of the Hessian sweep takes, and the shape that goes with them: threads, ring slots (a
// slot is 40 x 20 floats = 25 x 128 bytes) and blocks per SM.
template <int ROWS>
struct HessT {
  static constexpr int NT = kHTX / 4 * kHTY / ROWS;
  static constexpr int RING = ROWS == 2 ? 6 : 8;
  static constexpr size_t SMEM = (size_t)RING * kHPX * kHPY * 4 + (2 * RING) * 8 + (size_t)(NT / 32) * kHStage * sizeof(FgEntry);
};

// Input slices of the DoG sweep in flight: slice it + kDogIn - 1 is requested while slice it
// is filtered (2, 3 and 4 measured the same on the camera stack; 2 keeps the buffer index a
// bit mask).
#ifndef HDOG_DOG_STAGES
#define HDOG_DOG_STAGES 2
#endif
constexpr int kDogIn = HDOG_DOG_STAGES;

// ROWS: rows of the tile's columns a thread takes through the y pass and the z register.  The y pass reads 2R + ROWS
// x-filtered values for ROWS outputs from shared memory and the x pass filters 2R halo rows for a tile of NT / 32 * ROWS,
// so with two rows (a 32 x 16 tile, 80 registers, three blocks of 256 per SM) the shared-memory pipe was the limit (73%);
// four rows (32 x 24, 138 registers, two blocks of 192) leave it at 58% and the issue slots at 59%.  1.42 G voxels of
// radii (4, 6, 3, 5) 6.30 -> 5.63 ms, 0.71 G of (8, 12, 4, 5) 5.30 -> 4.29 ms.  Three rows (5.84 ms), five (6.07), one
// copy of the code for all z phases (6.37) and x pairs instead of scale pairs in the x pass (6.8) were slower.
template <int RA, int RB, int ZA, int ZB, int ROWS>
struct DogT {
  static constexpr int RXY = RA > RB ? RA : RB;
  static constexpr int RZ = ZA > ZB ? ZA : ZB;
  static constexpr int WIN = 2 * RZ + 1;
  static constexpr int NT = ROWS == 4 ? 192 : 256, BLOCKS = ROWS == 4 ? 2 : 3;
  static constexpr int TY = NT / kDTX * ROWS;                 // tile height
  static constexpr int HX = (RXY + 3) / 4 * 4;                // x halo, 16-byte aligned
  static constexpr int BW = kDTX + 2 * HX;                    // staged input box
  static constexpr int BH = TY + 2 * RXY;
  static constexpr int IN_FLOATS = (BW * BH + 31) / 32 * 32;  // 128-byte multiple
  static constexpr int XQ = kDTX / 4;                         // x-pass items of four outputs per row
  static constexpr int XITEMS = BH * XQ;
  static constexpr int NV = (HX + RXY + 4 + 3) / 4 * 4;       // inputs of an item, from column 4q
  static constexpr size_t SMEM = (size_t)kDogIn * IN_FLOATS * 4 + (size_t)2 * BH * kDTX * 8 + 8 * kDogIn + 64;
};

// Coefficient pairs (small, large) of the taps both scales share, |j| <= min(RA, RB),
// held in registers for the whole sweep: an f32x2 FMA takes its operands from registers,
// so pairs re-read from the constant bank would cost a load each use.  Taps of the
// wider scale alone stay constant-bank operands of scalar FMAs.
template <int RA, int RB>
struct TapPairs {
  static constexpr int RS = RA < RB ? RA : RB;
  static constexpr int N = RS + 1;
  float2 k[N];   // pair |j|: the taps are symmetric
  // The pairs as written by stage(): read back from shared memory, they are per-thread
  // registers, so the f32x2 FMAs use them directly instead of copying each pair out of
  // the uniform registers a kernel-parameter value would live in.
  __device__ __forceinline__ static void stage(const DogTaps &T, int ka, int kb, float2 *sh) {
#pragma unroll
    for (int j = 0; j <= RS; j++) sh[j] = make_float2(T.k[ka][RA - j], T.k[kb][RB - j]);
  }
  __device__ __forceinline__ void load_shared(const float2 *sh) {
#pragma unroll
    for (int i = 0; i < N; i++) k[i] = sh[i];
  }
};

// One tap of both scales: j is the input offset, the coefficient index r - j as in the
// reference's `sum = fma(k[r - j], s[x + j], sum)`.
template <int RA, int RB, int J>
__device__ __forceinline__ void tap2(const DogTaps &T, const TapPairs<RA, RB> &K, int ka, int kb, float2 v,
                                     float2 &acc) {
  constexpr bool a = J >= -RA && J <= RA, b = J >= -RB && J <= RB;
  if (a && b) acc = fma2(K.k[J < 0 ? -J : J], v, acc);
  else if (b) acc.y = __fmaf_rn(T.k[kb][RB - J], v.y, acc.y);
  else if (a) acc.x = __fmaf_rn(T.k[ka][RA - J], v.x, acc.x);
}

// x pass input by input: staged input w[I] is tap I - BASE - o of output o (o = 0..3), so its
// duplicated pair (one value for both scales of an f32x2 FMA) is formed once and used by up
// to four consecutive FMAs.  Every output still takes its taps in ascending order.
template <int RA, int RB, int BASE, int I, int NV>
struct XIn {
  __device__ __forceinline__ static void run(const DogTaps &T, const TapPairs<RA, RB> &K, const float (&w)[NV],
                                             float2 (&a)[4]) {
    if constexpr (I < NV) {
      const float2 d = make_float2(w[I], w[I]);
      tap2<RA, RB, I - BASE>(T, K, 0, 2, d, a[0]);
      tap2<RA, RB, I - BASE - 1>(T, K, 0, 2, d, a[1]);
      tap2<RA, RB, I - BASE - 2>(T, K, 0, 2, d, a[2]);
      tap2<RA, RB, I - BASE - 3>(T, K, 0, 2, d, a[3]);
      XIn<RA, RB, BASE, I + 1, NV>::run(T, K, w, a);
    }
  }
};

// y pass of ROWS rows, input row by input row: row I is tap I - R - o of output row o, read once, and every
// output still takes its taps in ascending order.
template <int RA, int RB, int ROWS, int I, int N>
struct YIn {
  static constexpr int R = RA > RB ? RA : RB;
  template <int O>
  __device__ __forceinline__ static void taps(const DogTaps &T, const TapPairs<RA, RB> &K, float2 v, float2 (&g)[ROWS]) {
    if constexpr (O < ROWS) {
      if constexpr (I - R - O >= -R && I - R - O <= R) tap2<RA, RB, I - R - O>(T, K, 0, 2, v, g[O]);
      taps<O + 1>(T, K, v, g);
    }
  }
  __device__ __forceinline__ static void run(const DogTaps &T, const TapPairs<RA, RB> &K, const float2 *col,
                                             float2 (&g)[ROWS]) {
    if constexpr (I < N) {
      taps<0>(T, K, col[I * kDTX], g);
      YIn<RA, RB, ROWS, I + 1, N>::run(T, K, col, g);
    }
  }
};

// z step of phase P = zy mod WIN: input slice zy is tap d of output zo = zy - d, which
// lives in slot (zo mod WIN); then output zy - RZ is complete and its slot is cleared for
// output zy - RZ + WIN.
template <class C, int ZA, int ZB, int ROWS, int P, int D0, int N>
struct ZTaps {
  __device__ __forceinline__ static void run(const DogTaps &T, const TapPairs<ZA, ZB> &K, float2 (&a)[ROWS][C::WIN],
                                             const float2 (&g)[ROWS]) {
    if constexpr (N > 0) {
      constexpr int s = ((P - D0) % C::WIN + C::WIN) % C::WIN;
#pragma unroll
      for (int o = 0; o < ROWS; o++) tap2<ZA, ZB, D0>(T, K, 1, 3, g[o], a[o][s]);
      ZTaps<C, ZA, ZB, ROWS, P, D0 + 1, N - 1>::run(T, K, a, g);
    }
  }
};

template <class C, int ZA, int ZB, int ROWS, int P>
__device__ __forceinline__ void z_step(const DogTaps &T, const TapPairs<ZA, ZB> &K, float2 (&a)[ROWS][C::WIN],
                                       const float2 (&g)[ROWS], float (&d)[ROWS]) {
  ZTaps<C, ZA, ZB, ROWS, P, -C::RZ, C::WIN>::run(T, K, a, g);
  constexpr int se = ((P - C::RZ) % C::WIN + C::WIN) % C::WIN;
#pragma unroll
  for (int o = 0; o < ROWS; o++) {
    d[o] = __fmul_rn(__fsub_rn(a[o][se].x, a[o][se].y), T.normalizer);
    a[o][se] = make_float2(0.f, 0.f);
  }
}

// Calls f(base + P, integral_constant<P>) for P = 0 .. N-1 while base + P < limit (the
// bound is uniform over the block, so every thread runs the same steps).
template <int P, int N, class F>
__device__ __forceinline__ void unroll_steps_from(F &f, int base, int limit) {
  if constexpr (P < N) {
    if (base + P < limit) {
      f(base + P, std::integral_constant<int, P>{});
      unroll_steps_from<P + 1, N>(f, base, limit);
    }
  }
}
template <int N, class F>
__device__ __forceinline__ void unroll_steps(F &f, int base, int limit) {
  unroll_steps_from<0, N>(f, base, limit);
}

// PERSIST: a grid of a few blocks per SM takes (substack, tile) items from the device work
// queue `q` until it is empty; otherwise one block per tile (blockIdx.x) and substack
// (blockIdx.y).  Results are the same either way.
template <int RA, int RB, int ZA, int ZB, int ROWS, bool PERSIST>
__global__ void __launch_bounds__(DogT<RA, RB, ZA, ZB, ROWS>::NT, DogT<RA, RB, ZA, ZB, ROWS>::BLOCKS)
    k_dog_sweep(const __grid_constant__ CUtensorMap map, const __grid_constant__ DogTaps T, const Sub *subs,
                float *dog, int *status, WorkQueue q) {
  using C = DogT<RA, RB, ZA, ZB, ROWS>;
  extern __shared__ __align__(128) unsigned char smem[];
  float *inb = reinterpret_cast<float *>(smem);
  float2 *xb = reinterpret_cast<float2 *>(inb + kDogIn * C::IN_FLOATS);   // two x-filtered slices, both scales
  uint64_t *bar = reinterpret_cast<uint64_t *>(xb + 2 * C::BH * kDTX);
  const int t = threadIdx.x;
  __shared__ float2 tap_sh[TapPairs<RA, RB>::N + TapPairs<ZA, ZB>::N];
  __shared__ int s_item;
  if (t == 0) {
    for (int i = 0; i < kDogIn; i++) mbar_init(&bar[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    TapPairs<RA, RB>::stage(T, 0, 2, tap_sh);
    TapPairs<ZA, ZB>::stage(T, 1, 3, tap_sh + TapPairs<RA, RB>::N);
  }
  bool ok = true;
  // slices loaded by this block before the current tile: slice `it` of a tile is the block's
  // (gbase + it)-th, which picks its input buffer (g mod kDogIn) and barrier phase
  uint32_t gbase = 0;
  for (;;) {
  int sub, tile;
  __syncthreads();   // the previous tile is done with both input buffers
  if (PERSIST) {
    if (t == 0) s_item = (int)atomicAdd(q.next, 1u);
    __syncthreads();
    const int item = s_item;
    if (item >= q.total) break;
    sub = item / q.tiles;
    tile = item % q.tiles;
  } else {
    sub = blockIdx.y;
    tile = blockIdx.x;
  }
  const Sub S = subs[sub];
  const int ntx = (S.W + kDTX - 1) / kDTX, nty = (S.H + C::TY - 1) / C::TY;
  if (tile >= ntx * nty) {
    if (PERSIST) continue;
    break;
  }
  const int x0 = (tile % ntx) * kDTX, y0 = (tile / ntx) * C::TY;
  const int D = S.D, W = S.W, H = S.H;
  constexpr uint32_t tma_bytes = (uint32_t)(C::BW * C::BH * 4);
  const int tx = x0 - C::HX, ty = y0 - C::RXY;
  if (t == 0 && ok)
    for (int z = 0; z < kDogIn - 1 && z < D; z++) {
      const uint32_t g = gbase + (uint32_t)z;
      tma_slice(&map, inb + (g % kDogIn) * C::IN_FLOATS, &bar[g % kDogIn], tx, ty, z, sub, tma_bytes);
    }
  // stage B ownership: columns (cx, cy .. cy + ROWS - 1) of the tile
  const int cx = t % kDTX, cy = ROWS * (t / kDTX);
  const int gx = x0 + cx, gy = y0 + cy;
  const float2 *yin = xb + cy * kDTX + cx;
  const int nrow = gx < W ? H - gy : 0;   // rows of them inside the frame
  float *out0 = dog + S.pvox + (int64_t)gy * S.P + gx;
  const int64_t WH = (int64_t)S.P * H;
  float2 acc[ROWS][C::WIN];
#pragma unroll
  for (int o = 0; o < ROWS; o++)
#pragma unroll
    for (int s = 0; s < C::WIN; s++) acc[o][s] = make_float2(0.f, 0.f);
  TapPairs<RA, RB> kxy;
  TapPairs<ZA, ZB> kz;
  kxy.load_shared(tap_sh);
  kz.load_shared(tap_sh + TapPairs<RA, RB>::N);
  const int nit = D + C::RZ + 1;
  // One slice step; PC is the step's position inside a group of WIN steps, so the z phase
  // of slice zy = it - 1 is the compile-time (PC - 1) mod WIN and every shift-register slot
  // is a fixed register (the loop below runs WIN steps per trip).
  auto step = [&](int it, auto PC) {
    constexpr int PH = (decltype(PC)::value + C::WIN - 1) % C::WIN;
    // slice it + kDogIn - 1 goes to the buffer of slice it - 1, read before the last barrier
    const uint32_t gn = gbase + (uint32_t)(it + kDogIn - 1);
    if (t == 0 && ok && it + kDogIn - 1 < D)
      tma_slice(&map, inb + (gn % kDogIn) * C::IN_FLOATS, &bar[gn % kDogIn], tx, ty, it + kDogIn - 1, sub, tma_bytes);
    // ---- B: y pass of slice zy (zero past the volume: the border taps still multiply),
    // z shift register, DoG slice zy - RZ
    const int zy = it - 1;
    if (zy >= 0) {
      float2 g[ROWS];
#pragma unroll
      for (int o = 0; o < ROWS; o++) g[o] = make_float2(0.f, 0.f);
      if (zy < D)
        YIn<RA, RB, ROWS, 0, 2 * C::RXY + ROWS>::run(T, kxy, yin + (zy & 1) * C::BH * kDTX, g);
      float d[ROWS];
      z_step<C, ZA, ZB, ROWS, PH>(T, kz, acc, g, d);
      const int zo = zy - C::RZ;
      if (zo >= 0) {
#pragma unroll
        for (int o = 0; o < ROWS; o++)
          if (o < nrow) out0[zo * WH + o * S.P] = d[o];
      }
    }
    // ---- A: x pass of slice it
    if (it < D) {
      const uint32_t gi = gbase + (uint32_t)it;
      if (ok && !mbar_wait(&bar[gi % kDogIn], (gi / kDogIn) & 1)) {
        ok = false;
        atomicExch(status, HDOG_ERR_TIMEOUT);
      }
      const float *ib = inb + (gi % kDogIn) * C::IN_FLOATS;
      float2 *xo = xb + (it & 1) * C::BH * kDTX;
      for (int item = t; item < C::XITEMS; item += (C::XITEMS <= C::NT ? C::XITEMS : C::NT)) {
        const int row = item / C::XQ, q = item % C::XQ;
        const float *in = ib + row * C::BW + 4 * q;
        float w[C::NV];
#pragma unroll
        for (int i = 0; i < C::NV; i += 4) {
          const float4 f = *reinterpret_cast<const float4 *>(in + i);
          w[i] = f.x; w[i + 1] = f.y; w[i + 2] = f.z; w[i + 3] = f.w;
        }
        float4 *o = reinterpret_cast<float4 *>(xo + row * kDTX + 4 * q);
        float2 a[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        XIn<RA, RB, C::HX, 0, C::NV>::run(T, kxy, w, a);
        o[0] = make_float4(a[0].x, a[0].y, a[1].x, a[1].y);
        o[1] = make_float4(a[2].x, a[2].y, a[3].x, a[3].y);
      }
    }
    __syncthreads();
  };
  for (int base = 0; base < nit; base += C::WIN)
    unroll_steps<C::WIN>(step, base, nit);
  gbase += (uint32_t)D;
  if (!PERSIST) break;
  }
}

// Central difference of the Hessian stage.  The reference writes ((0 + a) - b) * 0.5; the
// `0 +` only turns -0 into +0, and a zero's sign never changes a magnitude, a comparison
// or a fixed-point sum, so the mask and every record stay identical without it.
__device__ __forceinline__ float hdiff(float plus, float minus) { return __fmul_rn(__fsub_rn(plus, minus), 0.5f); }
// The same on two voxels at once (each lane rounds as the scalar operations do).
__device__ __forceinline__ float2 hd2(float2 plus, float2 minus) {
  return mul2(sub2(plus, minus), make_float2(0.5f, 0.5f));
}

// The pinned Sylvester test (common.cuh pd_test) on two voxels: every product and FMA is
// the scalar one lane by lane; fma(-(a*b), c, t) is written fma(a*b, c * -1, t), the same
// exact product with the sign moved.  Returns the two results in bits 0 and 8.
__device__ __forceinline__ uint32_t pd_test2(float2 xx, float2 xy, float2 xz, float2 yy, float2 yz, float2 zz) {
  const float2 m1 = make_float2(-1.0f, -1.0f);
  const float2 p = mul2(xx, yy);
  const float2 q = mul2(mul2(make_float2(2.0f, 2.0f), xy), yz);
  float2 t = fma2(p, zz, mul2(q, xz));
  t = fma2(mul2(xx, yz), mul2(yz, m1), t);
  t = fma2(mul2(yy, xz), mul2(xz, m1), t);
  const float2 xy2 = mul2(xy, xy);
  const float2 rhs = mul2(mul2(zz, xy), xy);
  const uint32_t a = (xx.x < 0.0f) & (p.x > xy2.x) & (t.x < rhs.x);
  const uint32_t b = (xx.y < 0.0f) & (p.y > xy2.y) & (t.y < rhs.y);
  return a | (b << 8);
}

// Gradient pairs of one ring row.  Voxel pairs come in two frames: the C frame
// (X0, X0+1), (X0+2, X0+3) -- the thread's own quad -- and the G frame (X0-1, X0),
// (X0+1, X0+2), (X0+3, X0+4), in which x differences of pairs loaded on 8-byte
// boundaries land without repacking.  gx in the G frame from the row's columns
// X0-2 .. X0+5 (l = X0-2, X0-1; c = the quad; r = X0+4, X0+5).
__device__ __forceinline__ void gx_g(float2 l, float2 c0, float2 c1, float2 r, float2 (&g)[3]) {
  g[0] = hd2(c0, l);
  g[1] = hd2(c1, c0);
  g[2] = hd2(r, c1);
}

__device__ __forceinline__ void ld_row(const float *p, float2 &l, float2 &c0, float2 &c1, float2 &r) {
  l = *reinterpret_cast<const float2 *>(p - 2);
  const float4 c = *reinterpret_cast<const float4 *>(p);
  c0 = make_float2(c.x, c.y);
  c1 = make_float2(c.z, c.w);
  r = *reinterpret_cast<const float2 *>(p + 4);
}
__device__ __forceinline__ void ld_quad(const float *p, float2 &c0, float2 &c1) {
  const float4 c = *reinterpret_cast<const float4 *>(p);
  c0 = make_float2(c.x, c.y);
  c1 = make_float2(c.z, c.w);
}


// Moves a warp's `n` staged entries to the substack's list: one slot reservation, then
// each lane completes whole entries -- the normalized value at the entry's voxel is
// gathered here, once per flush rather than on every slice -- and stores them as
// consecutive 32-byte entries.  Entries past the list's capacity are dropped but counted,
// so the host sees the overflow and redoes the batch.
template <bool PAD>
__device__ __forceinline__ void flush_stage(const FgEntry *stage, int n, const Sub &S, const float *norm, FgEntry *fg,
                                            int32_t *fg_idx, unsigned long long *count) {
  __syncwarp();
  const int lane = threadIdx.x & 31;
  unsigned long long base = 0;
  if (lane == 0) base = atomicAdd(count, (unsigned long long)n);
  base = __shfl_sync(0xFFFFFFFFu, base, 0);
  const int64_t room = S.fg_cap - (int64_t)base;
  const int keep = room <= 0 ? 0 : (room < n ? (int)room : n);
  const float *nv = norm + (PAD ? S.pvox : S.vox);
  const int extra = S.P - S.W;   // PAD: rows of the normalized volume are padded by this much
  // every lane's gathers are issued before any of them is used, so a flush waits for one
  // global-load latency rather than one per entry
  constexpr int kPer = kHStage / 32;
  int32_t idx[kPer];
  float nvv[kPer];
#pragma unroll
  for (int u = 0; u < kPer; u++) {
    const int i = lane + 32 * u;
    idx[u] = i < keep ? stage[i].idx : 0;
    nvv[u] = i < keep ? __ldg(nv + (PAD ? idx[u] + (int64_t)(idx[u] / S.W) * extra : idx[u])) : 0.0f;
  }
#pragma unroll
  for (int u = 0; u < kPer; u++) {
    const int i = lane + 32 * u;
    if (i < keep) {
      const float4 *src = reinterpret_cast<const float4 *>(stage + i);
      float4 a = src[0];
      a.y = nvv[u];
      float4 *dst = reinterpret_cast<float4 *>(fg + S.fg + base + i);
      dst[0] = a;
      dst[1] = src[1];
      fg_idx[S.fg + base + i] = idx[u];
    }
  }
  __syncwarp();
}

// PERSIST: a grid of a few blocks per SM takes (substack, tile) items from the device work
// queue `q` until it is empty; otherwise one block per tile (blockIdx.x) and substack
// (blockIdx.y).  SPLIT: the latter, with zlen slices per block (blockIdx.z) where the tiles alone leave most of
// the chip idle (a block's slices follow one another).  One 128x96x16 substack 28 -> 12 us, one of 256x256x32 63 ->
// 30 us.  Results are the same either way.  PAD: the width is no multiple of 4, so the rows of the
// DoG and the normalized volume are padded and the mask's are not whole words.
// ROWS 2: the two rows share the rows around them, 16 shared-memory reads and 32 wavefronts a row instead of 13 and
// 52, in 128 registers; 1.42 G voxels 5.11 -> 4.60 ms.  Blocks are half as wide in threads and take a slice as long,
// so batches without four waves of them keep one row (128x96x16: 12 us against 20; twelve small substacks: 155 against 187).
template <bool PERSIST, bool PAD, bool SPLIT, int ROWS>
__global__ void __launch_bounds__(HessT<ROWS>::NT, ROWS == 2 ? 7 : SPLIT ? 4 : 5)
    k_hess_sweep(const __grid_constant__ CUtensorMap map, const Sub *subs, const float *norm, uint8_t *mask,
                 FgEntry *fg, int32_t *fg_idx, unsigned long long *fg_count, int *status, WorkQueue q, int zlen) {
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int PL = kHPX * kHPY, RING = HessT<ROWS>::RING;
  constexpr uint32_t tma_bytes = (uint32_t)(PL * 4);
  float *ring = reinterpret_cast<float *>(smem);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem + (size_t)RING * PL * 4);
  // done[i % RING] completes when every warp has finished the block's i-th iteration, with
  // its last reads of that iteration's DoG slice zh-2
  uint64_t *done = bar + RING;
  const int t = threadIdx.x;
  // this warp's staging of list entries (flushed to the global list kHStage at a time at most)
  FgEntry *stage = reinterpret_cast<FgEntry *>(smem + (size_t)RING * PL * 4 + 2 * RING * 8) + (t >> 5) * kHStage;
  __shared__ int s_item;
  if (t == 0) {
    for (int i = 0; i < RING; i++) mbar_init(&bar[i], 1);
    for (int i = 0; i < RING; i++) mbar_init(&done[i], HessT<ROWS>::NT / 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  bool ok = true;
  // slices loaded into the ring and iterations run by this block before the current tile:
  // every tile loads its slices -2 .. D+1 once and runs D iterations, so the barrier phases
  // continue from tile to tile
  uint32_t zbase = 0, ibase = 0;
  for (;;) {
  int sub, tile;
  __syncthreads();   // every warp is done with the previous tile's ring slots
  if (PERSIST) {
    if (t == 0) s_item = (int)atomicAdd(q.next, 1u);
    __syncthreads();
    const int item = s_item;
    if (item >= q.total) break;
    sub = item / q.tiles;
    tile = item % q.tiles;
  } else {
    sub = blockIdx.y;
    tile = blockIdx.x;
  }
  const Sub S = subs[sub];
  const int ntx = (S.W + kHTX - 1) / kHTX, nty = (S.H + kHTY - 1) / kHTY;
  if (tile >= ntx * nty) {
    if (PERSIST) continue;
    break;
  }
  const int x0 = (tile % ntx) * kHTX, y0 = (tile / ntx) * kHTY;
  int staged = 0;   // entries in this warp's staging buffer (the same in every lane)
  const int D = S.D, W = S.W, H = S.H;
  const int32_t WH = W * H;
  const int tx = x0 - 4, ty = y0 - 2;
  const int zb = SPLIT ? (int)blockIdx.z * zlen : 0, ze = SPLIT ? min(D, zb + zlen) : D;   // this block's slices
  // ring slot of DoG slice z (z = zb-2 .. ze+1; slices outside the volume arrive zero-filled)
  auto slot = [zbase, zb](int z) { return (int)((zbase + (uint32_t)(z - zb + 2)) % RING); };
  // use k of slot s (k-th slice loaded into it) completes barrier phase k & 1
  auto use = [zbase, zb](int z) { return (int)((zbase + (uint32_t)(z - zb + 2)) / RING); };
  // the ring's slices but one up front, then slice zh + RING - 3 while slice zh is tested: the slot it
  // reuses held slice zh - 3, last read one iteration earlier
  if (t == 0 && ok)
    for (int z = zb - 2; z <= zb + RING - 4 && z <= ze + 1; z++)
      tma_slice(&map, ring + slot(z) * PL, &bar[slot(z)], tx, ty, z, sub, tma_bytes);
  for (int z = zb - 2; z <= zb + 1; z++)
    if (ok && !mbar_wait(&bar[slot(z)], use(z) & 1)) {
      ok = false;
      atomicExch(status, HDOG_ERR_TIMEOUT);
    }
  const int q = t % (kHTX / 4), ly = ROWS * (t / (kHTX / 4));
  const int X0 = x0 + 4 * q, Y = y0 + ly;      // the quad's column and first row
  const int b = (ly + 2) * kHPX + 4 * q + 4;   // ring index of column X0 on row Y
  // every in-plane gradient position of the quads inside the volume: the z-pipelined
  // stencil below (only the z neighbours can fall outside); the frame's edges take the
  // literal zero-halo path voxel by voxel.  Fixed per thread for the whole sweep.
  const bool interior = X0 >= 1 && X0 + 3 <= W - 2 && Y >= 1 && Y + ROWS <= H - 1;
  // z pipeline of the interior path, per row: first derivatives of slices zh-1 and zh
  // (gx in the G frame, gy and gz in the C frame) and DoG of slices zh and zh+1
  const float2 zero2 = make_float2(0.0f, 0.0f);
  float2 gxm[ROWS][3], gx0[ROWS][3], gym[ROWS][2], gy0[ROWS][2], fm[ROWS][2], f0[ROWS][2];
#pragma unroll
  for (int r = 0; r < ROWS; r++) {
    gxm[r][0] = gxm[r][1] = gxm[r][2] = zero2;
    gym[r][0] = gym[r][1] = zero2;
  }
  if (interior) {
    // slice zb: gx, gy on the thread's rows
    auto first = [&](const float *P, float2 (&gx)[ROWS][3], float2 (&gy)[ROWS][2], float2 (&c)[ROWS][2]) {
      float2 l, rr, u[2], d[2];
#pragma unroll
      for (int r = 0; r < ROWS; r++) {
        ld_row(P + r * kHPX, l, c[r][0], c[r][1], rr);
        gx_g(l, c[r][0], c[r][1], rr, gx[r]);
      }
      ld_quad(P - kHPX, u[0], u[1]);
      ld_quad(P + ROWS * kHPX, d[0], d[1]);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        gy[0][j] = hd2(ROWS == 2 ? c[ROWS - 1][j] : d[j], u[j]);
        if (ROWS == 2) gy[ROWS - 1][j] = hd2(d[j], c[0][j]);
      }
    };
    first(ring + slot(zb) * PL + b, gx0, gy0, fm);
    const float *P1 = ring + slot(zb + 1) * PL + b;
#pragma unroll
    for (int r = 0; r < ROWS; r++) ld_quad(P1 + r * kHPX, f0[r][0], f0[r][1]);
    if (SPLIT && zb > 0) {   // a block that starts inside the volume: the derivatives of slice zb-1 as well
      float2 c[ROWS][2];
      first(ring + slot(zb - 1) * PL + b, gxm, gym, c);
    }
  }
  for (int zh = zb; zh < ze; zh++) {
    // DoG slice zh+RING-3 reuses the slot of slice zh-3, read for the last time in iteration
    // zh-1: the producer waits until every warp is past it (warps otherwise run up to the
    // ring's depth apart)
    const int zn = zh + RING - 3;
    if (t == 0 && ok && zn <= ze + 1) {
      const uint32_t prev = ibase + (uint32_t)(zh - zb) - 1u;
      if (zh > zb && !mbar_wait(&done[prev % RING], (prev / RING) & 1)) {
        ok = false;
        atomicExch(status, HDOG_ERR_TIMEOUT);
      }
      if (ok) tma_slice(&map, ring + slot(zn) * PL, &bar[slot(zn)], tx, ty, zn, sub, tma_bytes);
    }
    // slices zh-2 .. zh+1 were waited for already; zh+2 is new
    if (ok && !mbar_wait(&bar[slot(zh + 2)], use(zh + 2) & 1)) {
      ok = false;
      atomicExch(status, HDOG_ERR_TIMEOUT);
    }
    const int32_t i0 = zh * WH + Y * W + X0;
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
      uint32_t mword = 0;
      float hv[4][6];
      const int32_t ir = i0 + r * W;
      if (interior) {
        // row 1 comes after row 0's advance: row 0's derivatives of slice zh are gxm[0] and gym[0] then, its DoG of
        // slice zh+1 is fm[0]
        const float *P0 = ring + slot(zh) * PL + b + r * kHPX, *P1 = ring + slot(zh + 1) * PL + b + r * kHPX;
        float2 hxx[2], hxy[3], hyy[2], hxz[3], hyz[2], hzz[2], gxp[3], gyp[2], fp[2], l, rr, c[2], e[2];
        hxx[0] = hd2(gx0[r][1], gx0[r][0]);
        hxx[1] = hd2(gx0[r][2], gx0[r][1]);
        // ---- in-plane second derivatives: the row beyond this one and the other row's first derivatives
        {
          float2 g[3];
          ld_row(r == 0 ? P0 - kHPX : P0 + kHPX, l, c[0], c[1], rr);
          gx_g(l, c[0], c[1], rr, g);
          ld_quad(r == 0 ? P0 - 2 * kHPX : P0 + 2 * kHPX, e[0], e[1]);
          if constexpr (ROWS == 2) {
#pragma unroll
            for (int i = 0; i < 3; i++) hxy[i] = r == 0 ? hd2(gx0[ROWS - 1][i], g[i]) : hd2(g[i], gxm[0][i]);
#pragma unroll
            for (int j = 0; j < 2; j++)
              hyy[j] = r == 0 ? hd2(gy0[ROWS - 1][j], hd2(fm[0][j], e[j])) : hd2(hd2(e[j], fm[r][j]), gym[0][j]);
          } else {
            float2 gd[3], k[2];
            ld_row(P0 + kHPX, l, c[0], c[1], rr);
            gx_g(l, c[0], c[1], rr, gd);
            ld_quad(P0 + 2 * kHPX, k[0], k[1]);
#pragma unroll
            for (int i = 0; i < 3; i++) hxy[i] = hd2(gd[i], g[i]);
#pragma unroll
            for (int j = 0; j < 2; j++) hyy[j] = hd2(hd2(k[j], fm[r][j]), hd2(fm[r][j], e[j]));
          }
        }
        // ---- first derivatives of slice zh+1, then the z second derivatives
        l = *reinterpret_cast<const float2 *>(P1 - 2);
        rr = *reinterpret_cast<const float2 *>(P1 + 4);
        gx_g(l, f0[r][0], f0[r][1], rr, gxp);
        ld_quad(r == 0 ? P1 - kHPX : P1 + kHPX, c[0], c[1]);
        float2 d[2];
        if (ROWS == 1) ld_quad(P1 + kHPX, d[0], d[1]);
        ld_quad(ring + slot(zh + 2) * PL + b + r * kHPX, fp[0], fp[1]);
        ld_quad(ring + slot(zh - 2) * PL + b + r * kHPX, e[0], e[1]);
        const bool zin = zh + 1 < D, zim = zh >= 1;   // gz outside the volume is zero
#pragma unroll
        for (int j = 0; j < 2; j++) {
          gyp[j] = ROWS == 1 ? hd2(d[j], c[j]) : r == 0 ? hd2(f0[ROWS - 1][j], c[j]) : hd2(c[j], fm[0][j]);
          hyz[j] = hd2(gyp[j], gym[r][j]);
          hzz[j] = hd2(zin ? hd2(fp[j], fm[r][j]) : zero2, zim ? hd2(fm[r][j], e[j]) : zero2);
        }
#pragma unroll
        for (int i = 0; i < 3; i++) hxz[i] = hd2(gxp[i], gxm[r][i]);
        // advance the pipeline
#pragma unroll
        for (int i = 0; i < 3; i++) { gxm[r][i] = gx0[r][i]; gx0[r][i] = gxp[i]; }
#pragma unroll
        for (int j = 0; j < 2; j++) {
          gym[r][j] = gy0[r][j]; gy0[r][j] = gyp[j];
          fm[r][j] = f0[r][j]; f0[r][j] = fp[j];
        }
        // G frame -> C frame for the two elements that live there (voxel 2j+h)
        const float2 cxy[2] = {make_float2(hxy[0].y, hxy[1].x), make_float2(hxy[1].y, hxy[2].x)};
        const float2 cxz[2] = {make_float2(hxz[0].y, hxz[1].x), make_float2(hxz[1].y, hxz[2].x)};
#pragma unroll
        for (int j = 0; j < 2; j++) {
          mword |= pd_test2(hxx[j], cxy[j], cxz[j], hyy[j], hyz[j], hzz[j]) << (16 * j);
          hv[2 * j][0] = hxx[j].x; hv[2 * j + 1][0] = hxx[j].y;
          hv[2 * j][1] = cxy[j].x; hv[2 * j + 1][1] = cxy[j].y;
          hv[2 * j][2] = cxz[j].x; hv[2 * j + 1][2] = cxz[j].y;
          hv[2 * j][3] = hyy[j].x; hv[2 * j + 1][3] = hyy[j].y;
          hv[2 * j][4] = hyz[j].x; hv[2 * j + 1][4] = hyz[j].y;
          hv[2 * j][5] = hzz[j].x; hv[2 * j + 1][5] = hzz[j].y;
        }
        uint8_t *mo = mask + S.vox + ir;
        if (!PAD) {
          *reinterpret_cast<uint32_t *>(mo) = mword;
        } else {   // the mask's rows are not padded
#pragma unroll
          for (int o = 0; o < 4; o++) mo[o] = (uint8_t)(mword >> (8 * o));
        }
      } else {
        const int yr = Y + r;
        const bool ym = yr >= 1, yp = yr + 1 < H, zm = zh >= 1, zp = zh + 1 < D;
        const int br = b + r * kHPX;
        const int p0 = slot(zh) * PL + br, p1 = slot(zh + 1) * PL + br, p2 = slot(zh + 2) * PL + br;
        const int m1 = slot(zh - 1) * PL + br, m2 = slot(zh - 2) * PL + br;
#pragma unroll
        for (int o = 0; o < 4; o++) {
          const int X = X0 + o;
          if (X >= W || yr >= H) continue;
          // the slices hold zeros outside the volume, so a first derivative only needs the zero of its own
          // position outside: past the frame's sides (xm .. yp) or the first and last slice (zm, zp)
          const bool xm = X >= 1, xp = X + 1 < W;
          const float *c0 = ring + p0 + o, *cu = ring + p1 + o, *cd = ring + m1 + o;
          hv[o][0] = hdiff(xp ? hdiff(c0[2], c0[0]) : 0.0f, xm ? hdiff(c0[0], c0[-2]) : 0.0f);
          hv[o][1] = hdiff(yp ? hdiff(c0[kHPX + 1], c0[kHPX - 1]) : 0.0f, ym ? hdiff(c0[1 - kHPX], c0[-1 - kHPX]) : 0.0f);
          hv[o][2] = hdiff(zp ? hdiff(cu[1], cu[-1]) : 0.0f, zm ? hdiff(cd[1], cd[-1]) : 0.0f);
          hv[o][3] = hdiff(yp ? hdiff(c0[2 * kHPX], c0[0]) : 0.0f, ym ? hdiff(c0[0], c0[-2 * kHPX]) : 0.0f);
          hv[o][4] = hdiff(zp ? hdiff(cu[kHPX], cu[-kHPX]) : 0.0f, zm ? hdiff(cd[kHPX], cd[-kHPX]) : 0.0f);
          hv[o][5] = hdiff(zp ? hdiff(ring[p2 + o], c0[0]) : 0.0f, zm ? hdiff(c0[0], ring[m2 + o]) : 0.0f);
          const bool pdv = pd_test(hv[o][0], hv[o][1], hv[o][2], hv[o][3], hv[o][4], hv[o][5]);
          mask[S.vox + ir + o] = pdv ? 1 : 0;
          // voxel 0 is background (its label is 0 in the reference's CCL)
          mword |= (pdv && ir + o != 0 ? 1u : 0u) << (8 * o);
        }
      }
      // the foreground voxels go to the warp's staging buffer in shared memory; a full buffer
      // goes to the global list with one slot reservation and coalesced stores (and the
      // entries' normalized values).  Warps without foreground skip all of it; each lane's
      // place comes from three bit-sliced ballots of its count.
      const int nfg = __popc(mword);
      const unsigned any = __ballot_sync(0xFFFFFFFFu, nfg != 0);
      if (any) {
        const int lane = t & 31;
        const unsigned b0 = __ballot_sync(0xFFFFFFFFu, nfg & 1), b1 = __ballot_sync(0xFFFFFFFFu, nfg & 2),
                       b2 = __ballot_sync(0xFFFFFFFFu, nfg & 4);
        const unsigned lt = (1u << lane) - 1u;
        const int excl = __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
        const int tot = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
        if (staged + tot > kHStage) {
          flush_stage<PAD>(stage, staged, S, norm, fg, fg_idx, &fg_count[sub * kFgCountStride]);
          staged = 0;
        }
        int k = staged + excl;
#pragma unroll
        for (int o = 0; o < 4; o++) {
          if (!((mword >> (8 * o)) & 1u)) continue;
          float4 *dst = reinterpret_cast<float4 *>(stage + k);
          dst[0] = make_float4(__int_as_float(ir + o), 0.0f, hv[o][0], hv[o][1]);
          dst[1] = make_float4(hv[o][2], hv[o][3], hv[o][4], hv[o][5]);
          k++;
        }
        staged += tot;
      }
    }
    __syncwarp();
    if ((t & 31) == 0) mbar_arrive(&done[(ibase + (uint32_t)(zh - zb)) % RING]);
  }
  if (staged) flush_stage<PAD>(stage, staged, S, norm, fg, fg_idx, &fg_count[sub * kFgCountStride]);
  zbase += (uint32_t)(D + 4);
  ibase += (uint32_t)D;
  if (!PERSIST) break;
  }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Radius-specialised instantiations: (small xy, large xy, small z, large z) tap radii.
// (4, 6, 3, 5): sigma (2.0, 1.5) / (3.2, 2.4); (8, 12, 4, 5): sigma (4.0, 1.8) / (6.0, 2.7).
typedef void (*DogSweepKernel)(CUtensorMap, DogTaps, const Sub *, float *, int *, WorkQueue);
struct SweepForm {
  DogSweepKernel fn, fn_persist;
  size_t smem;
  int threads, ty, bw, bh;
};
struct SweepInst {
  int ra, rb, za, zb;
  SweepForm form[2];   // two and four rows per thread
};
template <int RA, int RB, int ZA, int ZB, int ROWS>
constexpr SweepForm sweep_form() {
  using C = DogT<RA, RB, ZA, ZB, ROWS>;
  return SweepForm{k_dog_sweep<RA, RB, ZA, ZB, ROWS, false>, k_dog_sweep<RA, RB, ZA, ZB, ROWS, true>,
                   C::SMEM, C::NT, C::TY, C::BW, C::BH};
}
template <int RA, int RB, int ZA, int ZB>
constexpr SweepInst sweep_inst() {
  return SweepInst{RA, RB, ZA, ZB, {sweep_form<RA, RB, ZA, ZB, 2>(), sweep_form<RA, RB, ZA, ZB, 4>()}};
}
static const SweepInst kSweepInst[] = {sweep_inst<4, 6, 3, 5>(), sweep_inst<8, 12, 4, 5>()};

// The sweep for these taps, or none.  The four-row form where its 32 x 24 tiles give every SM its two blocks; below
// that the two-row form's smaller ones, whose blocks take a slice sooner (one 128x96x16 substack 11.9 against 13.9 us).
// A wave of either covers as many voxels (two blocks of 24 rows, three of 16), the four-row one in 0.81 to 0.89 of the
// time, so heights that fill the 24-row tiles badly, or start another wave of them, stay with 16 rows.  us, 24 / 16
// rows, radii (4, 6, 3, 5), 8 slices: 70000x8 75/57, 10000x32 29/23, 4000x100 29/26, 10000x40 30/30; 16 slices of
// 4000x112 48/43, of 2560x2160 389/420.
static const SweepForm *find_form(const DogTaps &T, int W, int H, int nsub, int num_sms) {
  for (const SweepInst &s : kSweepInst)
    if (s.ra == T.r[0] && s.rb == T.r[2] && s.za == T.r[1] && s.zb == T.r[3]) {
      const int64_t cols = (int64_t)ceil_div(W, kDTX) * nsub;
      const int64_t tall = cols * ceil_div(H, s.form[1].ty), flat = cols * ceil_div(H, s.form[0].ty);
      const auto waves = [](int64_t tiles, int64_t room) { return 0.5 * ((double)tiles / room + (double)((tiles + room - 1) / room)); };
      return &s.form[tall >= 2 * (int64_t)num_sms && 0.85 * waves(tall, 2 * num_sms) <= waves(flat, 3 * num_sms)];
    }
  return nullptr;
}

static_assert((kHPX * kHPY * 4) % 128 == 0, "TMA ring slots must start on 128-byte boundaries");

// Whether the Hessian sweep can run at all (its volumes are the context's own, padded for TMA).
bool sweep_supported(int max_smem) { return encode_fn() != nullptr && (int)HessT<1>::SMEM <= max_smem; }

static CUresult encode_map(CUtensorMap *map, const float *base, int W, int P, int H, int D, int nsub, int bw, int bh) {
  if (encode_fn() == nullptr) return CUDA_ERROR_NOT_SUPPORTED;
  const cuuint64_t dims[4] = {(cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)D, (cuuint64_t)nsub};
  const cuuint64_t strides[3] = {(cuuint64_t)P * 4, (cuuint64_t)P * H * 4, (cuuint64_t)P * H * D * 4};
  const cuuint32_t box[4] = {(cuuint32_t)bw, (cuuint32_t)bh, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(base), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

// One launch of a radius-specialised DoG sweep: a block per tile and substack, or (per_sm > 0)
// per_sm blocks per SM over the work queue whose counter is *qctr (zero at the launch).
static void dog_sweep_launch(const SweepForm *si, const CUtensorMap &map_n, const DogTaps &T, const Sub *d_subs,
                             int nsub, int W, int H, float *dog, int *d_status, const LaunchShape &ls,
                             unsigned *qctr, cudaStream_t s) {
  const unsigned tiles_d = ceil_div(W, kDTX) * ceil_div(H, si->ty);
  if (ls.dog_per_sm > 0 && qctr) {
    const WorkQueue q{qctr, (int)(tiles_d * (unsigned)nsub), (int)tiles_d};
    const unsigned grid = std::min<unsigned>((unsigned)(ls.dog_per_sm * ls.num_sms), tiles_d * (unsigned)nsub);
    cudaFuncSetAttribute(si->fn_persist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)si->smem);
    KLAUNCH("k_dog_sweep", s, (si->fn_persist<<<grid, si->threads, si->smem, s>>>(map_n, T, d_subs, dog, d_status, q)));
    return;
  }
  cudaFuncSetAttribute(si->fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)si->smem);
  KLAUNCH("k_dog_sweep", s, (si->fn<<<dim3(tiles_d, nsub), si->threads, si->smem, s>>>(map_n, T, d_subs, dog, d_status,
                                                                                        WorkQueue{})));
}

bool launch_dog_sweep(const Sub *d_subs, int nsub, int W, int P, int H, int D, const DogTaps &T, const float *norm,
                      float *dog, int *d_status, int max_smem, cudaStream_t s) {
  const SweepForm *si = find_form(T, W, H, nsub, LaunchShape{}.num_sms);
  if (!si || P % 4 != 0 || (int)si->smem > max_smem || encode_fn() == nullptr) return false;
  if ((reinterpret_cast<uintptr_t>(norm) & 15) != 0) return false;
  CUtensorMap map_n;
  if (encode_map(&map_n, norm, W, P, H, D, nsub, si->bw, si->bh) != CUDA_SUCCESS) return false;
  dog_sweep_launch(si, map_n, T, d_subs, nsub, W, H, dog, d_status, LaunchShape{}, nullptr, s);
  return true;
}

int launch_dog_hess(const Sub *d_subs, int nsub, int W, int P, int H, int D, const DogTaps &T, const float *norm,
                    float2 *fa, float2 *fb, float *dog, uint8_t *mask, FgEntry *fg, int32_t *fg_idx,
                    unsigned long long *fg_count, int *d_status, const LaunchShape &ls, unsigned *qctr, int max_smem,
                    cudaStream_t s) {
  const SweepForm *si = find_form(T, W, H, nsub, ls.num_sms);
  CUtensorMap map_n, map_d;
  if (encode_map(&map_d, dog, W, P, H, D, nsub, kHPX, kHPY) != CUDA_SUCCESS) return HDOG_ERR_CUDA;
  if (si && (int)si->smem <= max_smem && encode_map(&map_n, norm, W, P, H, D, nsub, si->bw, si->bh) == CUDA_SUCCESS)
    dog_sweep_launch(si, map_n, T, d_subs, nsub, W, H, dog, d_status, ls, qctr, s);
  else
    launch_dog(d_subs, nsub, W, P, H, D, (int64_t)H * D, T, norm, fa, fb, dog, s);
  const unsigned tiles_h = ceil_div(W, kHTX) * ceil_div(H, kHTY);
  if (ls.hess_per_sm > 0 && qctr) {
    const WorkQueue q{qctr + 1, (int)(tiles_h * (unsigned)nsub), (int)tiles_h};
    const unsigned grid = std::min<unsigned>((unsigned)(ls.hess_per_sm * ls.num_sms), tiles_h * (unsigned)nsub);
    auto fn = P != W ? k_hess_sweep<true, true, false, 1> : k_hess_sweep<true, false, false, 1>;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)HessT<1>::SMEM);
    KLAUNCH("k_hess_sweep", s, (fn<<<grid, HessT<1>::NT, HessT<1>::SMEM, s>>>(map_d, d_subs, norm, mask, fg, fg_idx, fg_count,
                                                                      d_status, q, D)));
  } else {
    // split z while the blocks about fit the chip at once (four per SM, and half as many again while those run), down
    // to six slices: a piece spends about two slices' time on the four it loads around its own.  256x256x32 alone: one
    // piece 63 us, five 30 us; 683x517x75, whose tiles fill the chip, 221 us unsplit
    const int64_t room = (int64_t)6 * ls.num_sms / ((int64_t)tiles_h * nsub);
    const int pieces = (int)std::max<int64_t>(1, std::min<int64_t>(room, D / 6)), zlen = (int)ceil_div(D, pieces);
    const bool two = (int64_t)tiles_h * nsub >= 28 * (int64_t)ls.num_sms;   // four waves of seven blocks per SM
    auto fn = two        ? (P != W ? k_hess_sweep<false, true, false, 2> : k_hess_sweep<false, false, false, 2>)
              : zlen < D ? (P != W ? k_hess_sweep<false, true, true, 1> : k_hess_sweep<false, false, true, 1>)
                         : (P != W ? k_hess_sweep<false, true, false, 1> : k_hess_sweep<false, false, false, 1>);
    const unsigned nt = two ? HessT<2>::NT : HessT<1>::NT;
    const size_t smem = two ? HessT<2>::SMEM : HessT<1>::SMEM;
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    KLAUNCH("k_hess_sweep", s, (fn<<<dim3(tiles_h, nsub, ceil_div(D, zlen)), nt, smem, s>>>(
                                   map_d, d_subs, norm, mask, fg, fg_idx, fg_count, d_status, WorkQueue{}, zlen)));
  }
  return HDOG_OK;
}

}  // namespace hdog
