// soft.cu -- the differentiable HDoG chain, sm_103a: forward and hand-written adjoint of
// normalize -> DoG -> Hessian -> relaxed positive-definiteness score at sample points.
//
// Forward stages follow the reference's (NormalizeFilter.cu:537-654, DoG3DFilter.cu:70-437,
// Hessian3DFilter_element.cu:22-388) with its borders, in float32 without the bit-exact
// summation orders of the detection path: min / max and box means with nearest borders,
// separable Gaussians with zero borders (one sigma per axis and scale), central
// differences of central differences with zeros outside the volume, and the mask test
// xx < 0, xx yy - xy^2 > 0, det < 0 relaxed to a product of sigmoids of the minors scaled
// by tau, tau^2, tau^3.  Loss = mean score at the positive points - mean score at the
// negative points.
//
// With few sample points the DoG, its derivatives and the transposed Gaussians are evaluated at the
// points' neighbourhoods (k_soft_points_local); with many, over the volume as follows.
//
// Backward recomputes every intermediate from the input, or (the _kept entry) takes the
// forward chain's intermediates from the workspace the forward call filled, which the
// backward does not overwrite, and runs the adjoints in reverse: the score's derivative scattered through the
// Hessian stencil into a DoG-shaped gradient; for the sigmas, the derivative-of-Gaussian
// taps (d t_k / d sigma = t_k (k^2 - sum_j t_j j^2) / sigma^3 for the normalized taps) on
// one axis and the plain taps on the others, dotted with that gradient, plus the
// normalizer's term; for the input, the transposed separable Gaussians (the taps are
// symmetric and the borders zero, so the transpose is the same correlation), the
// normalization's quotient rule, the transposed box means (a gather that counts how often
// the nearest border repeats each edge value) and the transposed min / max filters (each
// window's gradient goes to its first extreme, recomputed from the filter's input).
// Tap radii are (int)(2 sigma + 0.5), held fixed for the derivatives.
//
#include <algorithm>
#include <climits>
#include <cmath>

#include "kernels.cuh"
#include "window.cuh"

namespace hdog {

constexpr int kSoftMaxRadius = 31;
constexpr int kSoftMaxTaps = 2 * kSoftMaxRadius + 1;
struct SoftTaps {
  float k[kSoftMaxTaps];
  int r;
};
struct SoftGeom {
  int W, H, D;
};

__device__ __forceinline__ void soft_axis(const SoftGeom &g, int axis, int64_t i, int &c, int64_t &stride, int &n) {
  const int x = (int)(i % g.W), y = (int)((i / g.W) % g.H), z = (int)(i / ((int64_t)g.W * g.H));
  if (axis == 0) { c = x; stride = 1; n = g.W; }
  else if (axis == 1) { c = y; stride = g.W; n = g.H; }
  else { c = z; stride = (int64_t)g.W * g.H; n = g.D; }
}

// One separable Gaussian pass (zero border) from a shared-memory tile: a block stages the inputs of
// its outputs once (along x a row segment of kSoftTileX outputs plus the taps' reach on each side;
// along y or z a 32-column slab of kSoftTileYZ outputs plus the reach), zero outside the line, and every
// output folds its taps in ascending order, skipping those outside the line.
constexpr int kSoftTileX = 256, kSoftTileYZ = 64;

__device__ __forceinline__ float soft_fold(const float *w, int step, int c, int n, const SoftTaps &T) {
  // w[k * step] is the input at line position c - T.r + k
  float acc = 0.0f;
  for (int j = -T.r; j <= T.r; j++) {
    const int p = c + j;
    if (p >= 0 && p < n) acc = __fmaf_rn(T.k[j + T.r], w[(j + T.r) * step], acc);
  }
  return acc;
}

__device__ __forceinline__ float soft_stage(const float *line, int64_t s, int p, int n) {
  return (p >= 0 && p < n) ? line[(int64_t)p * s] : 0.0f;
}

// Dot products as compensated float32 sums (GB300's FP64 pipe is a small fraction of its
// FP32 rate): a product a b is split exactly into p + e (p = a b rounded, e = fma(a, b, -p)),
// added to a running hi + lo by Knuth's TwoSum (the rounding error of hi + p goes to lo), and
// per warp the pairs combine the same way before one conversion to double; the relative error
// of a thread's or warp's sum is about 2^-48, against 2^-53 per addition of a double sum.
__device__ __forceinline__ void soft_two_sum(float &hi, float &lo, float v) {
  const float s = __fadd_rn(hi, v), bb = __fsub_rn(s, hi);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bb)), __fsub_rn(v, bb)));
  hi = s;
}

__device__ __forceinline__ void soft_dot_add(float &hi, float &lo, float a, float b) {
  const float p = __fmul_rn(a, b);
  lo = __fadd_rn(lo, __fmaf_rn(a, b, -p));
  soft_two_sum(hi, lo, p);
}

// the warp's (hi, lo) pairs summed into lane 0's, returned as a double there
__device__ __forceinline__ double soft_warp_dot(float hi, float lo) {
  for (int o = 16; o > 0; o >>= 1) {
    const float h2 = __shfl_down_sync(0xFFFFFFFFu, hi, o), l2 = __shfl_down_sync(0xFFFFFFFFu, lo, o);
    lo = __fadd_rn(lo, l2);
    soft_two_sum(hi, lo, h2);
  }
  return (double)hi + (double)lo;
}

// along x: a block takes the same segment of kSoftRowsX consecutive rows (so each thread has
// several loads in flight before the barrier), one output per thread and row
constexpr int kSoftRowsX = 4;

__global__ void __launch_bounds__(kSoftTileX) k_soft_pass_x(const float *in, float *out, SoftGeom g, SoftTaps T,
                                                            const unsigned *skip) {
  if (skip && *skip) return;   // the output is already there
  __shared__ float tile[kSoftRowsX][kSoftTileX + 2 * kSoftMaxRadius];
  const int nseg = (g.W + kSoftTileX - 1) / kSoftTileX;
  const int64_t row0 = (int64_t)(blockIdx.x / nseg) * kSoftRowsX;
  const int nr = (int)min((int64_t)kSoftRowsX, (int64_t)g.H * g.D - row0);
  const int x0 = (int)(blockIdx.x % nseg) * kSoftTileX, t = threadIdx.x;
  const int L = kSoftTileX + 2 * T.r;
  for (int r = 0; r < nr; r++)
    for (int k = t; k < L; k += kSoftTileX) tile[r][k] = soft_stage(in + (row0 + r) * g.W, 1, x0 - T.r + k, g.W);
  __syncthreads();
  const int x = x0 + t;
  if (x < g.W)
    for (int r = 0; r < nr; r++) out[(row0 + r) * g.W + x] = soft_fold(tile[r] + t, 1, x, g.W, T);
}

// along y (AXIS 1) or z (AXIS 2): a block of 32 x 8 threads owns 32 columns and
// kSoftTileYZ outputs of each; thread (tx, ty) computes outputs ty, ty + 8, ...  The epilogue
// stores the outputs (kEpiStore); or stores scale * (aux - output), the DoG difference
// (kEpiDiff); or stores nothing and adds sum(output * aux) over the block's outputs to
// *dot_out (kEpiDot; a double, from compensated float32 sums up to the warps).
enum { kEpiStore = 0, kEpiDot = 1, kEpiDiff = 2 };

template <int AXIS, int EPI = kEpiStore>
__global__ void __launch_bounds__(256) k_soft_pass_yz(const float *in, float *out, SoftGeom g, SoftTaps T,
                                                      const unsigned *skip = nullptr,
                                                      const float *aux = nullptr, double *dot_out = nullptr,
                                                      float scale = 0.0f) {
  if (skip && *skip) return;
  extern __shared__ float slab[];   // [kSoftTileYZ + 2R][32]
  const int tx = threadIdx.x, ty = threadIdx.y, R = T.r;
  const int n = AXIS == 1 ? g.H : g.D;
  const int64_t s = AXIS == 1 ? (int64_t)g.W : (int64_t)g.W * g.H;
  const int x = blockIdx.x * 32 + tx;
  const int c0 = blockIdx.y * kSoftTileYZ;
  // the other coordinate: z for the y pass, y for the z pass
  const int64_t other = AXIS == 1 ? (int64_t)blockIdx.z * g.W * g.H : (int64_t)blockIdx.z * g.W;
  const float *line = in + other + x;
  const int rows = kSoftTileYZ + 2 * R;
  for (int k = ty; k < rows; k += 8) slab[k * 32 + tx] = x < g.W ? soft_stage(line, s, c0 - R + k, n) : 0.0f;
  __syncthreads();
  float hi = 0.0f, lo = 0.0f;
  if (x < g.W)
    for (int m = ty; m < kSoftTileYZ; m += 8) {
      const int c = c0 + m;
      if (c >= n) break;
      const int64_t i = other + x + (int64_t)c * s;
      const float v = soft_fold(slab + m * 32 + tx, 32, c, n, T);
      if (EPI == kEpiDot) soft_dot_add(hi, lo, aux[i], v);
      else if (EPI == kEpiDiff) out[i] = scale * (aux[i] - v);
      else out[i] = v;
    }
  if (EPI == kEpiDot) {
    __shared__ double part[8];
    const double acc = soft_warp_dot(hi, lo);
    if (tx == 0) part[ty] = acc;
    __syncthreads();
    if (tx == 0 && ty == 0) {
      double t = 0.0;
      for (int w = 0; w < 8; w++) t += part[w];
      atomicAdd(dot_out, t);
    }
  }
}

// ---- normalization windows: min and max (and their box means) travel as one float2 per voxel
//
// All passes handle both sides at once, so a volume is read and written once per axis.  Extremes come
// from short blocks (window.cuh); their adjoints find each window's first extreme the same way, every
// combination taking a later entry only when it is strictly better, and a thread adds up the gradients
// of its consecutive windows with one extreme before the atomic add.  Box means fold each output's
// window from 0 in ascending order (the sigma gradients are sensitive to the last bits of the
// normalized volume), K neighbouring outputs per thread from a rotating register window.  Reaches that
// the rings or tiles do not hold take the *_far kernels, which read each window from global memory; below a
// block (r < 4) the row passes take them too, the column passes fold their windows in registers (*_short).
struct MinMaxF {
  typedef float2 T;
  __device__ __forceinline__ static float2 op(float2 a, float2 b) { return make_float2(fminf(a.x, b.x), fmaxf(a.y, b.y)); }
};

// A window's first min and first max, and their entries.
struct ExtAt {
  float2 v;
  int a, b;
};
// the extremes of a span and of one after it (or overlapping its end)
__device__ __forceinline__ ExtAt ext_join(const ExtAt &p, const ExtAt &q) {
  ExtAt r = p;
  if (q.v.x < p.v.x) {
    r.v.x = q.v.x;
    r.a = q.a;
  }
  if (q.v.y > p.v.y) {
    r.v.y = q.v.y;
    r.b = q.b;
  }
  return r;
}

// Adds the gradients of consecutive windows that share their extreme (the entries never decrease along
// a line) and puts each run's sum where the extreme lies.
template <class PutF>
struct RunSum {
  int at = -1;
  float sum = 0.0f;
  PutF put;
  __device__ __forceinline__ RunSum(PutF p) : put(p) {}
  __device__ __forceinline__ void add(int a, float g) {
    if (a != at) {
      flush();
      at = a;
      sum = 0.0f;
    }
    sum += g;
  }
  __device__ __forceinline__ void flush() {
    if (sum != 0.0f) put(at, sum);
  }
};

// Line geometry of a pass along y (AXIS 1) or z (AXIS 2): block x = 32 columns, block y = the other coordinate.
template <int AXIS>
struct SoftLine {
  int n, x;
  int64_t base, s;
  bool in;
  __device__ __forceinline__ SoftLine(const SoftGeom &g) {
    n = AXIS == 1 ? g.H : g.D;
    s = AXIS == 1 ? (int64_t)g.W : (int64_t)g.W * g.H;
    x = blockIdx.x * 32 + threadIdx.x;
    in = x < g.W;
    base = (AXIS == 1 ? (int64_t)blockIdx.y * g.W * g.H : (int64_t)blockIdx.y * g.W) + min(x, g.W - 1);
  }
};

constexpr int kSoftB = 8;   // block of the column passes

// min / max along y or z, segments of `seg` positions (blockIdx.z)
template <int AXIS, int NW>
__global__ void __launch_bounds__(32 * NW) k_soft_ext_cols(const float2 *in, float2 *out, SoftGeom g, int r, int seg) {
  extern __shared__ float2 ring2[];
  const SoftLine<AXIS> l(g);
  const int t0 = blockIdx.z * seg;
  ext_cols<MinMaxF, kSoftB, NW>(
      ring2, min(seg, l.n - t0), r,
      [&](int a, float2 (&v)[kSoftB]) {
#pragma unroll
        for (int j = 0; j < kSoftB; j++) v[j] = __ldg(in + l.base + (int64_t)clampi(t0 - r + a + j, 0, l.n - 1) * l.s);
      },
      [&](int t, float2 m) {
        if (l.in) out[l.base + (int64_t)(t0 + t) * l.s] = m;
      });
}

// The adjoint along y or z: src the pass's input, gout its output's gradient, added to gin (zeroed before).
// As ext_cols with the suffixes' places in their blocks kept beside them, but one warp per 32 columns
// runs down a segment alone: it needs no block barrier, and a run of windows with one extreme goes on from
// block to block, so that few voxels take an atomic add (interleaved blocks of 8 warps ended a run every
// 8 outputs).  The next block's inputs and gradients are loaded before this one is worked on.
// 512x512x128, reaches 20 and 5: y 244 -> 202 us, z 240 -> 150 us.
template <int AXIS>
__global__ void __launch_bounds__(32) k_soft_ext_adj_cols(const float2 *src, const float2 *gout, float2 *gin, SoftGeom g,
                                                          int r, int seg) {
  constexpr int B = kSoftB;
  extern __shared__ float2 ring2[];
  const SoftLine<AXIS> l(g);
  const int lane = threadIdx.x, t0 = blockIdx.z * seg, n = min(seg, l.n - t0);
  const int rows = ext_cols_rows(r, B, 1), total = n + 2 * r, back = (2 * r + B - 1) / B, q = back * B - 2 * r;
  uint16_t *place = reinterpret_cast<uint16_t *>(ring2 + rows * 32);
  float *gi = reinterpret_cast<float *>(gin);
  auto put = [&](int side) {
    return [=](int e, float v) {
      atomicAdd(gi + 2 * (l.base + (int64_t)clampi(t0 - r + e, 0, l.n - 1) * l.s) + side, v);
    };
  };
  RunSum<decltype(put(0))> lo(put(0)), hi(put(1));
  float2 nv[B], ng[B];
  auto fetch = [&](int a) {
    const int y = t0 - r + a;
    if (y >= 0 && y + B <= l.n) {
      const float2 *p = src + l.base + (int64_t)y * l.s;
#pragma unroll
      for (int j = 0; j < B; j++, p += l.s) nv[j] = __ldg(p);
    } else {
#pragma unroll
      for (int j = 0; j < B; j++) nv[j] = __ldg(src + l.base + (int64_t)clampi(y + j, 0, l.n - 1) * l.s);
    }
    if (a + B > 2 * r) {
#pragma unroll
      for (int j = 0; j < B; j++) ng[j] = __ldg(gout + l.base + (int64_t)clampi(t0 + a + j - 2 * r, 0, l.n - 1) * l.s);
    }
  };
  fetch(0);
  int pos = 0;
  for (int a = 0; a < total; a += B) {
    float2 v[B], go[B];
#pragma unroll
    for (int j = 0; j < B; j++) {
      v[j] = nv[j];
      go[j] = ng[j];
    }
    if (a + B < total) fetch(a + B);
    ExtAt s{v[B - 1], B - 1, B - 1};
#pragma unroll
    for (int j = B - 1; j >= 0; j--) {
      if (j < B - 1) s = ext_join(ExtAt{v[j], j, j}, s);
      ring2[(pos + j) * 32 + lane] = s.v;
      place[(pos + j) * 32 + lane] = (uint16_t)(s.a | s.b << 8);
    }
    if (a + B > 2 * r) {   // a lane reads its own column only
      auto row = [&](int d) {
        const int p = pos - d * B;
        return p < 0 ? p + rows : p;
      };
      auto get = [&](int p, int blk0) {   // ring row p, whose block starts at entry blk0
        const int k = place[p * 32 + lane];
        return ExtAt{ring2[p * 32 + lane], blk0 + (k & 0xFF), blk0 + (k >> 8)};
      };
      ExtAt mid1, mid0;
      if (back >= 3) {
        mid1 = get(row(back - 2), a - (back - 2) * B);
        for (int d = back - 3; d >= 1; d--) mid1 = ext_join(mid1, get(row(d), a - d * B));
      }
      if (back >= 2) {
        mid0 = get(row(back - 1), a - (back - 1) * B);
        if (back >= 3) mid0 = ext_join(mid0, mid1);
      }
      const int r0 = row(back), r1 = back >= 2 ? row(back - 1) : r0;
      ExtAt p{v[0], a, a};
#pragma unroll
      for (int o = 0; o < B; o++) {
        const int e = a + o;
        if (o) p = ext_join(p, ExtAt{v[o], e, e});
        if (e < 2 * r || e >= total) continue;
        const bool first = o < B - q;
        ExtAt m = first ? get(r0 + q + o, a - back * B) : get(r1 + q + o - B, a - (back - 1) * B);
        if (first ? back >= 2 : back >= 3) m = ext_join(m, first ? mid0 : mid1);
        m = ext_join(m, p);
        if (l.in) {
          lo.add(m.a, go[o].x);
          hi.add(m.b, go[o].y);
        }
      }
    }
    pos += B;
    if (pos >= rows) pos -= rows;
  }
  lo.flush();
  hi.flush();
}

// 32-byte global accesses where the address allows them (sm_100 on), else entry by entry
__device__ __forceinline__ void soft_ld8(const float *p, float (&v)[8]) {
  if ((reinterpret_cast<uintptr_t>(p) & 31) == 0) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
        : "l"(p));
  } else {
#pragma unroll
    for (int o = 0; o < 8; o++) v[o] = __ldg(p + o);
  }
}
__device__ __forceinline__ void soft_st8(float *p, const float (&v)[8]) {
  if ((reinterpret_cast<uintptr_t>(p) & 31) == 0) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
                 : "memory");
  } else {
#pragma unroll
    for (int o = 0; o < 8; o++) p[o] = v[o];
  }
}

// min / max along x of the volume itself, G lanes per row (window.cuh); rows start `pad` entries early
// so that a lane's eight outputs start on 32 bytes
constexpr int kSoftRowWarps = 4;

template <int G, int Q>
__global__ void __launch_bounds__(32 * kSoftRowWarps) k_soft_ext_rows(const float *in, float2 *out, SoftGeom g, int r) {
  using R = RowRing<G>;
  __shared__ float2 smr[kSoftRowWarps][R::WORDS];
  const int W = g.W, gl = threadIdx.x & (G - 1), w = threadIdx.x >> 5;
  const int64_t rows = (int64_t)g.H * g.D, row0 = ((int64_t)blockIdx.x * kSoftRowWarps + w) * R::LINES;
  if (row0 >= rows) return;
  const int64_t mine = row0 + (threadIdx.x & 31) / G, row = min(mine, rows - 1);
  const bool live = mine < rows;
  const float *line = in + row * W;
  float2 *o2 = out + row * W;
  // (for reaches that are multiples of 4 the inputs do too)
  const int pad = r % 4 == 0 ? (int)((reinterpret_cast<uintptr_t>(line - r) >> 2) & 7)
                             : (int)((reinterpret_cast<uintptr_t>(o2 - 2 * r) >> 3) & 3);
  const int n_in = W + 2 * r;
  float nv[8];
  float2 hist[6];
#pragma unroll
  for (int k = 0; k < 6; k++) hist[k] = make_float2(0.0f, 0.0f);
  auto fetch = [&](int c) {
    const int x = c + 8 * gl - r;
    if (x >= 0 && x + 8 <= W) {
      soft_ld8(line + x, nv);
    } else {
#pragma unroll
      for (int o = 0; o < 8; o++) nv[o] = __ldg(line + clampi(x + o, 0, W - 1));
    }
  };
  int c = -pad, pc = 0;
  fetch(c);
  for (int i = 0; i < n_in + 7; i += R::CHUNK, c += R::CHUNK) {
    float2 v[8], m[8];
#pragma unroll
    for (int o = 0; o < 8; o++) v[o] = make_float2(nv[o], nv[o]);
    if (i < n_in) fetch(c + R::CHUNK);
    ext_row_chunk<MinMaxF, G, Q>(smr[w], pc, r, v, hist, m);
    const int u = c + 8 * gl - 2 * r;
    if (live) {
      if (u >= 0 && u + 8 <= W) {
        const float a[8] = {m[0].x, m[0].y, m[1].x, m[1].y, m[2].x, m[2].y, m[3].x, m[3].y};
        const float b[8] = {m[4].x, m[4].y, m[5].x, m[5].y, m[6].x, m[6].y, m[7].x, m[7].y};
        soft_st8(reinterpret_cast<float *>(o2 + u), a);
        soft_st8(reinterpret_cast<float *>(o2 + u + 4), b);
      } else {
#pragma unroll
        for (int o = 0; o < 8; o++)
          if (u + o >= 0 && u + o < W) o2[u + o] = m[o];
      }
    }
    __syncwarp();
    pc += G;
    if (pc >= R::NB) pc = 0;
  }
}

template <int G>
__device__ __forceinline__ ExtAt row_lag_at(const ExtAt &cur, const ExtAt &prev, int lag) {
  return ExtAt{make_float2(row_lag<G>(cur.v.x, prev.v.x, lag), row_lag<G>(cur.v.y, prev.v.y, lag)),
               row_lag<G>(cur.a, prev.a, lag), row_lag<G>(cur.b, prev.b, lag)};
}

// The adjoint along x: both sides' gradients go to the volume's gradient gin, at the first min and first max of each
// window of the volume src.  As ext_row_chunk, with places.
template <int G, int Q>
__global__ void __launch_bounds__(32 * kSoftRowWarps) k_soft_ext_adj_rows(const float *src, const float2 *gout, float *gin,
                                                                          SoftGeom g, int r) {
  using R = RowRing<G>;
  __shared__ float2 smv[kSoftRowWarps][R::WORDS];
  __shared__ uint16_t smp[kSoftRowWarps][R::WORDS];
  const int W = g.W, gl = threadIdx.x & (G - 1), w = threadIdx.x >> 5;
  const int64_t rows = (int64_t)g.H * g.D, row0 = ((int64_t)blockIdx.x * kSoftRowWarps + w) * R::LINES;
  if (row0 >= rows) return;
  const int64_t mine = row0 + (threadIdx.x & 31) / G, row = min(mine, rows - 1);
  const bool live = mine < rows;
  const float *line = src + row * W;
  const float2 *go2 = gout + row * W;
  float *gi = gin + row * W;
  float2 *suf = smv[w];
  uint16_t *place = smp[w];
  const int pad = r % 4 == 0 ? (int)((reinterpret_cast<uintptr_t>(line - r) >> 2) & 7)
                             : (int)((reinterpret_cast<uintptr_t>(go2 - 2 * r) >> 3) & 3);
  const int n_in = W + 2 * r, back = (2 * r + 7) / 8, n1 = back - 2;
  float nv[8];
  ExtAt hist[6];
#pragma unroll
  for (int k = 0; k < 6; k++) hist[k] = ExtAt{make_float2(0.0f, 0.0f), 0, 0};
  auto fetch = [&](int c) {
    const int x = c + 8 * gl - r;
    if (x >= 0 && x + 8 <= W) {
      soft_ld8(line + x, nv);
    } else {
#pragma unroll
      for (int o = 0; o < 8; o++) nv[o] = __ldg(line + clampi(x + o, 0, W - 1));
    }
  };
  auto put = [=](int e, float v) { atomicAdd(gi + clampi(e - r, 0, W - 1), v); };
  int c = -pad, pc = 0;
  fetch(c);
  for (int i = 0; i < n_in + 7; i += R::CHUNK, c += R::CHUNK) {
    float v[8];
#pragma unroll
    for (int o = 0; o < 8; o++) v[o] = nv[o];
    if (i < n_in) fetch(c + R::CHUNK);
    const int e0 = c + 8 * gl, u = e0 - 2 * r;
    float2 go[8];
    if (u >= 0 && u + 8 <= W) {
      float a[8], b[8];
      soft_ld8(reinterpret_cast<const float *>(go2 + u), a);
      soft_ld8(reinterpret_cast<const float *>(go2 + u + 4), b);
#pragma unroll
      for (int o = 0; o < 4; o++) {
        go[o] = make_float2(a[2 * o], a[2 * o + 1]);
        go[4 + o] = make_float2(b[2 * o], b[2 * o + 1]);
      }
    } else {
#pragma unroll
      for (int o = 0; o < 8; o++) go[o] = u + o >= 0 && u + o < W ? __ldg(go2 + u + o) : make_float2(0.0f, 0.0f);
    }
    const RowAt<G> at(pc);
    const int own = at(0);
    ExtAt s{make_float2(v[7], v[7]), e0 + 7, e0 + 7};
#pragma unroll
    for (int o = 7; o >= 0; o--) {
      if (o < 7) s = ext_join(ExtAt{make_float2(v[o], v[o]), e0 + o, e0 + o}, s);
      suf[o * R::PITCH + own] = s.v;
      place[o * R::PITCH + own] = (uint16_t)((s.a - e0) | (s.b - e0) << 8);
    }
    __syncwarp();
    ExtAt mid1, mid0, d = s;
#pragma unroll
    for (int k = 0; k < (G == 8 ? 3 : 6); k++) {
      if ((1 << k) <= n1) {
        const bool last = (2 << k) > n1;
        if (last) mid1 = ext_join(row_lag_at<G>(d, hist[k], 1 + n1 - (1 << k)), row_lag_at<G>(d, hist[k], 1));
        const ExtAt h = hist[k];
        hist[k] = d;
        if (!last) d = ext_join(row_lag_at<G>(d, h, 1 << k), d);
      }
    }
    auto get = [&](int o, int b, int blk0) {
      const int k = place[o * R::PITCH + b];
      return ExtAt{suf[o * R::PITCH + b], blk0 + (k & 0xFF), blk0 + (k >> 8)};
    };
    const int b0 = at(back), b1 = at(back >= 2 ? back - 1 : 1);
    if (back >= 2) {
      mid0 = get(0, b1, e0 - 8 * (back - 1));
      if (n1 >= 1) mid0 = ext_join(mid0, mid1);
    }
    RunSum<decltype(put)> lo(put), hi(put);
    ExtAt p{make_float2(v[0], v[0]), e0, e0};
#pragma unroll
    for (int o = 0; o < 8; o++) {
      const int e = e0 + o;
      if (o) p = ext_join(p, ExtAt{make_float2(v[o], v[o]), e, e});
      ExtAt m;
      if (Q + o < 8) {
        m = get(Q + o, b0, e0 - 8 * back);
        if (back >= 2) m = ext_join(m, mid0);
      } else {
        m = get(Q + o - 8, b1, e0 - 8 * (back - 1));
        if (n1 >= 1) m = ext_join(m, mid1);
      }
      m = ext_join(m, p);
      if (live && u + o >= 0 && u + o < W) {
        lo.add(m.a, go[o].x);
        hi.add(m.b, go[o].y);
      }
    }
    lo.flush();
    hi.flush();
    __syncwarp();
    pc += G;
    if (pc >= R::NB) pc = 0;
  }
}

// One input of a box fold: clamped to the line (the mean), or zero outside it (ADJ, the transposed mean,
// whose edge outputs take the repeated edge taps on top).
__device__ __forceinline__ float2 soft_fma2(float k, float2 v, float2 a) {
  return make_float2(__fmaf_rn(k, v.x, a.x), __fmaf_rn(k, v.y, a.y));
}
// the extra taps of the transposed mean at the line's ends: output t's window ran past position 0 (n - 1) R - t
// (t + R - (n - 1)) times; ld(t): the gradient at t
template <class LoadF>
__device__ __forceinline__ float2 soft_box_ends(int c, int n, int R, LoadF ld, float2 acc) {
  if (c == 0)
    for (int t = 0; t < min(n, R); t++) acc = soft_fma2((float)(R - t), ld(t), acc);
  if (c == n - 1)
    for (int t = max(0, n - R); t < n; t++) acc = soft_fma2((float)(t + R - (n - 1)), ld(t), acc);
  return acc;
}
// the same for K outputs from c0 (a multiple of K) on: only the first of them can be the line's first, any its
// last, so each loop stands once in the code
template <int K, class LoadF>
__device__ __forceinline__ void soft_box_ends_k(int c0, int n, int R, LoadF ld, float2 (&acc)[K]) {
  if (c0 == 0)
    for (int t = 0; t < min(n, R); t++) acc[0] = soft_fma2((float)(R - t), ld(t), acc[0]);
  const int last = n - 1 - c0;
  if (last >= K) return;
  float2 e = acc[0];
#pragma unroll
  for (int k = 1; k < K; k++) e = k == last ? acc[k] : e;
  for (int t = max(0, n - R); t < n; t++) e = soft_fma2((float)(t + R - (n - 1)), ld(t), e);
#pragma unroll
  for (int k = 0; k < K; k++) acc[k] = k == last ? e : acc[k];
}

// Box mean along x (or its transpose): a tile of 32 rows x kSoftBoxX outputs with the reach on both sides in shared
// memory (odd pitch: a lane's row starts in its own bank), one row per lane and kSoftBoxK outputs per thread.
constexpr int kSoftBoxK = 16, kSoftBoxX = 128;

template <bool ADJ>
__global__ void __launch_bounds__(256, 2) k_soft_box_x(const float2 *in, float2 *out, SoftGeom g, int R) {
  extern __shared__ float2 tile2[];
  const int pitch = (kSoftBoxX + 2 * R) | 1, n0 = kSoftBoxX + 2 * R;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nseg = (g.W + kSoftBoxX - 1) / kSoftBoxX;
  const int64_t rows = (int64_t)g.H * g.D, row0 = (int64_t)(blockIdx.x / nseg) * 32;
  const int x0 = (int)(blockIdx.x % nseg) * kSoftBoxX, nr = (int)min((int64_t)32, rows - row0);
  for (int k = w; k < nr; k += 8) {
    const float2 *line = in + (row0 + k) * g.W;
    for (int i = lane; i < n0; i += 32) {
      const int x = x0 - R + i;
      // asynchronous, so that all of a thread's loads are in flight at once; outside the line (ADJ) no bytes, zeros
      const bool zero = ADJ && (x < 0 || x >= g.W);
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(tile2 + k * pitch + i)),
                   "l"(line + clampi(x, 0, g.W - 1)), "r"(zero ? 0 : 8)
                   : "memory");
    }
  }
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float2 acc[kSoftBoxK];
  const float2 *mine = tile2 + lane * pitch;
  const int xw = w * kSoftBoxK;
  const bool work = lane < nr && x0 + xw < g.W;
  if (work) {
    box_chain<kSoftBoxK>(2 * R + 1, [&](int i) { return mine[xw + i]; }, acc);
    if (ADJ) soft_box_ends_k(x0 + xw, g.W, R, [&](int t) { return mine[t - x0 + R]; }, acc);
    const SoftDiv div(2 * R + 1);
#pragma unroll
    for (int k = 0; k < kSoftBoxK; k++) acc[k] = div(acc[k]);
  }
  __syncthreads();
  if (work)
#pragma unroll
    for (int k = 0; k < kSoftBoxK; k++) tile2[lane * pitch + xw + k] = acc[k];
  __syncthreads();
  for (int k = w; k < nr; k += 8)
    for (int i = lane; i < min(kSoftBoxX, g.W - x0); i += 32) out[(row0 + k) * g.W + x0 + i] = tile2[k * pitch + i];
}

// Box mean along y or z (or its transpose), K outputs of one column per thread; NORM (z, the last
// pass): also the normalized volume, *bad set when a value of it is not finite (a window without contrast).
// RT: the reach where it is known at compile time (all of a thread's loads are then in flight before the
// first add), else 0.
template <int AXIS, int K, bool ADJ, bool NORM, int RT>
__global__ void __launch_bounds__(128) k_soft_box_cols(const float2 *in, float2 *out, SoftGeom g, int R_, const float *I,
                                                       float *norm, float min_intensity, unsigned *bad) {
  const SoftLine<AXIS> l(g);
  const int c0 = (blockIdx.z * blockDim.y + threadIdx.y) * K;
  if (!l.in || c0 >= l.n) return;
  const float2 *col = in + l.base;
  const int R = RT ? RT : R_;
  float2 acc[K];
  float iv[K];
  if (NORM) {
#pragma unroll
    for (int k = 0; k < K; k++) iv[k] = __ldg(I + l.base + (int64_t)min(c0 + k, l.n - 1) * l.s);
  }
  if constexpr (RT > 0) {
    float2 win[K + 2 * RT];
#pragma unroll
    for (int i = 0; i < K + 2 * RT; i++) {
      const int c = c0 - RT + i;
      win[i] = ADJ && (c < 0 || c >= l.n) ? make_float2(0.0f, 0.0f) : __ldg(col + (int64_t)clampi(c, 0, l.n - 1) * l.s);
    }
#pragma unroll
    for (int k = 0; k < K; k++) {
      acc[k] = make_float2(0.0f, 0.0f);
#pragma unroll
      for (int j = 0; j <= 2 * RT; j++) acc[k] = add2(acc[k], win[k + j]);
    }
  } else if (c0 - R >= 0 && c0 + K + R <= l.n) {
    const float2 *p = col + (int64_t)(c0 - R) * l.s;
    box_chain<K>(2 * R + 1, [&](int i) { return __ldg(p + (int64_t)i * l.s); }, acc);
  } else {
    box_chain<K>(2 * R + 1, [&](int i) {
      const int c = c0 - R + i;
      return ADJ && (c < 0 || c >= l.n) ? make_float2(0.0f, 0.0f) : __ldg(col + (int64_t)clampi(c, 0, l.n - 1) * l.s);
    }, acc);
  }
  if (ADJ) soft_box_ends_k(c0, l.n, R, [&](int t) { return __ldg(col + (int64_t)t * l.s); }, acc);
  const SoftDiv div(2 * R + 1);
#pragma unroll
  for (int k = 0; k < K; k++) {
    const int c = c0 + k;
    if (c >= l.n) break;
    const int64_t i = l.base + (int64_t)c * l.s;
    const float2 m = div(acc[k]);
    out[i] = m;
    if (NORM) {
      const float v = iv[k] >= min_intensity ? (iv[k] - m.x) / (m.y - m.x) : 0.0f;
      norm[i] = v;
      if (!isfinite(v)) *bad = 1u;
    }
  }
}

// Column passes below a block (r < 4): a warp takes kSoftShort outputs of 32 columns with their inputs in registers, so
// a window of up to seven costs a load an output instead of seven.  187x203x61 at reach 3: extremes 22.6 -> 5.8 us,
// adjoint 24.1 -> 12.0 us.
constexpr int kSoftShort = 8;
template <int AXIS, int R>
__global__ void __launch_bounds__(256) k_soft_ext_short(const float2 *in, float2 *out, SoftGeom g) {
  const SoftLine<AXIS> l(g);
  const int t0 = (blockIdx.z * 8 + threadIdx.y) * kSoftShort;
  if (t0 >= l.n || !l.in) return;
  float2 v[kSoftShort + 2 * R];
#pragma unroll
  for (int j = 0; j < kSoftShort + 2 * R; j++) v[j] = __ldg(in + l.base + (int64_t)clampi(t0 - R + j, 0, l.n - 1) * l.s);
#pragma unroll
  for (int k = 0; k < kSoftShort; k++) {
    float2 m = v[k];
#pragma unroll
    for (int j = 1; j <= 2 * R; j++) m = MinMaxF::op(m, v[k + j]);
    if (t0 + k < l.n) out[l.base + (int64_t)(t0 + k) * l.s] = m;
  }
}

template <int AXIS, int R>
__global__ void __launch_bounds__(256) k_soft_ext_adj_short(const float2 *src, const float2 *gout, float2 *gin, SoftGeom g) {
  const SoftLine<AXIS> l(g);
  const int t0 = (blockIdx.z * 8 + threadIdx.y) * kSoftShort;
  if (t0 >= l.n || !l.in) return;
  float *gi = reinterpret_cast<float *>(gin);
  auto put = [&](int side) {
    return [=](int e, float v) { atomicAdd(gi + 2 * (l.base + (int64_t)clampi(t0 - R + e, 0, l.n - 1) * l.s) + side, v); };
  };
  RunSum<decltype(put(0))> lo(put(0)), hi(put(1));
  float2 v[kSoftShort + 2 * R], go[kSoftShort];
#pragma unroll
  for (int j = 0; j < kSoftShort + 2 * R; j++) v[j] = __ldg(src + l.base + (int64_t)clampi(t0 - R + j, 0, l.n - 1) * l.s);
#pragma unroll
  for (int k = 0; k < kSoftShort; k++)
    go[k] = t0 + k < l.n ? __ldg(gout + l.base + (int64_t)(t0 + k) * l.s) : make_float2(0.0f, 0.0f);
#pragma unroll
  for (int k = 0; k < kSoftShort; k++) {
    if (t0 + k >= l.n) break;
    ExtAt m{v[k], k, k};
#pragma unroll
    for (int j = 1; j <= 2 * R; j++) m = ext_join(m, ExtAt{v[k + j], k + j, k + j});
    lo.add(m.a, go[k].x);
    hi.add(m.b, go[k].y);
  }
  lo.flush();
  hi.flush();
}

// Any reach, from global memory: the extremes of a line of float2 (or, FIRST, of the volume itself)
template <bool FIRST>
__device__ __forceinline__ float2 soft_far_ld(const void *p, int64_t i) {
  if (FIRST) {
    const float v = __ldg(static_cast<const float *>(p) + i);
    return make_float2(v, v);
  }
  return __ldg(static_cast<const float2 *>(p) + i);
}

template <bool FIRST>
__global__ void k_soft_ext_far(const void *in, float2 *out, SoftGeom g, int axis, int r, int64_t N) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int c, n;
  int64_t s;
  soft_axis(g, axis, i, c, s, n);
  const int64_t base = i - (int64_t)c * s;
  float2 m = soft_far_ld<FIRST>(in, i);
  for (int t = max(0, c - r); t <= min(n - 1, c + r); t++) m = MinMaxF::op(m, soft_far_ld<FIRST>(in, base + (int64_t)t * s));
  out[i] = m;
}

template <bool FIRST>
__global__ void k_soft_ext_adj_far(const void *src, const float2 *gout, float *gin, SoftGeom g, int axis, int r, int64_t N) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int c, n;
  int64_t s;
  soft_axis(g, axis, i, c, s, n);
  const int64_t base = i - (int64_t)c * s;
  const int t0 = max(0, c - r);
  ExtAt m{soft_far_ld<FIRST>(src, base + (int64_t)t0 * s), t0, t0};
  for (int t = t0 + 1; t <= min(n - 1, c + r); t++)
    m = ext_join(m, ExtAt{soft_far_ld<FIRST>(src, base + (int64_t)t * s), t, t});
  const float2 go = gout[i];
  const int step = FIRST ? 1 : 2;
  if (go.x != 0.0f) atomicAdd(gin + step * (base + (int64_t)m.a * s), go.x);
  if (go.y != 0.0f) atomicAdd(gin + step * (base + (int64_t)m.b * s) + step - 1, go.y);
}

// (sums of 753 values and more: compensated, a plain float32 chain that long is off by 1e-5 of a score)
template <bool ADJ>
__global__ void k_soft_box_far(const float2 *in, float2 *out, SoftGeom g, int axis, int R, int64_t N) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  int c, n;
  int64_t s;
  soft_axis(g, axis, i, c, s, n);
  const float2 *line = in + (i - (int64_t)c * s);
  float2 hi = make_float2(0.0f, 0.0f), lo = hi;
  for (int j = -R; j <= R; j++) {
    const int t = c + j;
    if (ADJ && (t < 0 || t >= n)) continue;
    const float2 v = line[(int64_t)clampi(t, 0, n - 1) * s];
    soft_two_sum(hi.x, lo.x, v.x);
    soft_two_sum(hi.y, lo.y, v.y);
  }
  float2 acc = add2(hi, lo);
  if (ADJ) acc = soft_box_ends(c, n, R, [&](int t) { return line[(int64_t)t * s]; }, acc);
  out[i] = SoftDiv(2 * R + 1)(acc);
}

// The normalized volume from the box means where no other pass forms it (see k_soft_box_cols).
__global__ void k_soft_norm(const float *I, const float2 *ed, float *norm, float min_intensity, int64_t N, unsigned *bad) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  const float iv = I[i];
  const float2 m = ed[i];
  const float v = iv >= min_intensity ? (iv - m.x) / (m.y - m.x) : 0.0f;
  norm[i] = v;
  if (!isfinite(v)) *bad = 1u;
}

// Quotient rule of the normalization: g_I (direct term, written) and the gradients of both box means.
__device__ __forceinline__ void soft_norm_adj_one(float v, float2 m, float g, float min_intensity, float &gi, float2 &ged) {
  if (v >= min_intensity) {
    const float den = m.y - m.x, inv = 1.0f / den, inv2 = inv * inv;
    gi = g * inv;
    ged = make_float2(g * (v - m.y) * inv2, -g * (v - m.x) * inv2);
  } else {
    gi = 0.0f;
    ged = make_float2(0.0f, 0.0f);
  }
}

// Four neighbouring gradients of the normalized volume
__device__ __forceinline__ float4 soft_ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float4 soft_ld4(const double *p) {
  const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
  return make_float4((float)a.x, (float)a.y, (float)b.x, (float)b.y);
}

// VEC 4: four voxels per thread in 16-byte accesses (I and g_I on 16 bytes; the workspace's volumes are).  g_norm in
// doubles may lie where g_ed goes: a voxel's eight bytes are read before they are written.
template <int VEC, class GT>
__global__ void __launch_bounds__(256) k_soft_norm_adj(const float *I, const float2 *ed, const GT *g_norm, float *g_I,
                                                       float2 *g_ed, float min_intensity, int64_t N) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (VEC == 4 && i + 4 <= N) {
    const float4 v = __ldg(reinterpret_cast<const float4 *>(I + i)), g = soft_ld4(g_norm + i);
    const float4 m0 = __ldg(reinterpret_cast<const float4 *>(ed + i)), m1 = __ldg(reinterpret_cast<const float4 *>(ed + i) + 1);
    float4 gi;
    float2 a, b, c, d;
    soft_norm_adj_one(v.x, make_float2(m0.x, m0.y), g.x, min_intensity, gi.x, a);
    soft_norm_adj_one(v.y, make_float2(m0.z, m0.w), g.y, min_intensity, gi.y, b);
    soft_norm_adj_one(v.z, make_float2(m1.x, m1.y), g.z, min_intensity, gi.z, c);
    soft_norm_adj_one(v.w, make_float2(m1.z, m1.w), g.w, min_intensity, gi.w, d);
    *reinterpret_cast<float4 *>(g_I + i) = gi;
    reinterpret_cast<float4 *>(g_ed + i)[0] = make_float4(a.x, a.y, b.x, b.y);
    reinterpret_cast<float4 *>(g_ed + i)[1] = make_float4(c.x, c.y, d.x, d.y);
    return;
  }
  for (int64_t k = i; k < min(i + VEC, N); k++) soft_norm_adj_one(I[k], ed[k], (float)g_norm[k], min_intensity, g_I[k], g_ed[k]);
}

// a += b.x + b.y (no window along any of x and y: both sides' gradients belong where they are)
__global__ void k_soft_add(float *a, const float2 *b, int64_t N) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) a[i] += b[i].x + b[i].y;
}

// sum_i a[i] * b[i] into *out (a double, which must start at zero; compensated float32 sums
// up to the warps)
__global__ void k_soft_dot(const float *a, const float *b, int64_t N, double *out) {
  __shared__ double part[8];
  float hi = 0.0f, lo = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (int64_t)gridDim.x * blockDim.x)
    soft_dot_add(hi, lo, a[i], b[i]);
  const double acc = soft_warp_dot(hi, lo);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += part[w];
    atomicAdd(out, t);
  }
}

// ---- Hessian at a point and its adjoint (element order xx, xy, xz, yy, yz, zz)
__device__ __forceinline__ int h_inner(int e) { return e < 3 ? 0 : (e < 5 ? 1 : 2); }   // xx xy xz | yy yz | zz
__device__ __forceinline__ int h_outer(int e) { return e == 0 ? 0 : (e == 1 || e == 3 ? 1 : 2); }

// Offsets of the three relaxed minor tests (kernel parameter).
struct SoftThresh {
  float v[3];
};

struct SoftPoint {
  int x, y, z;
};
__device__ __forceinline__ bool soft_in(const SoftGeom &g, int x, int y, int z) {
  return x >= 0 && y >= 0 && z >= 0 && x < g.W && y < g.H && z < g.D;
}
__device__ __forceinline__ void soft_step(int axis, int s, int &x, int &y, int &z) {
  if (axis == 0) x += s;
  else if (axis == 1) y += s;
  else z += s;
}
__device__ __forceinline__ float soft_f(const float *f, const SoftGeom &g, int x, int y, int z) {
  return soft_in(g, x, y, z) ? f[((int64_t)z * g.H + y) * g.W + x] : 0.0f;
}

__device__ void soft_hessian(const float *f, const SoftGeom &g, SoftPoint p, float h[6]) {
  for (int e = 0; e < 6; e++) {
    float v = 0.0f;
    for (int sb = -1; sb <= 1; sb += 2) {
      int qx = p.x, qy = p.y, qz = p.z;
      soft_step(h_outer(e), sb, qx, qy, qz);
      if (!soft_in(g, qx, qy, qz)) continue;   // a first derivative outside the volume is 0
      int ax = qx, ay = qy, az = qz, bx = qx, by = qy, bz = qz;
      soft_step(h_inner(e), 1, ax, ay, az);
      soft_step(h_inner(e), -1, bx, by, bz);
      const float ga = 0.5f * (soft_f(f, g, ax, ay, az) - soft_f(f, g, bx, by, bz));
      v += sb > 0 ? ga : -ga;
    }
    h[e] = 0.5f * v;
  }
}

// (in doubles: many points may meet in one voxel)
__device__ void soft_hessian_adj(double *gf, const SoftGeom &g, SoftPoint p, const float gh[6]) {
  for (int e = 0; e < 6; e++) {
    for (int sb = -1; sb <= 1; sb += 2) {
      int qx = p.x, qy = p.y, qz = p.z;
      soft_step(h_outer(e), sb, qx, qy, qz);
      if (!soft_in(g, qx, qy, qz)) continue;
      const float c = 0.25f * (float)sb * gh[e];
      int ax = qx, ay = qy, az = qz, bx = qx, by = qy, bz = qz;
      soft_step(h_inner(e), 1, ax, ay, az);
      soft_step(h_inner(e), -1, bx, by, bz);
      if (soft_in(g, ax, ay, az)) atomicAdd(gf + ((int64_t)az * g.H + ay) * g.W + ax, (double)c);
      if (soft_in(g, bx, by, bz)) atomicAdd(gf + ((int64_t)bz * g.H + by) * g.W + bx, -(double)c);
    }
  }
}

__device__ __forceinline__ float sigm(float v) { return 1.0f / (1.0f + expf(-v)); }

// Score of Hessian h: sigmoid((b0 - xx) / tau) sigmoid((m2 - b1) / tau^2) sigmoid((b2 - det) /
// tau^3) with thresholds b (all zero: the reference's test xx < 0, m2 > 0, det < 0).  When
// ds is given, its derivative in h; when db is given, its derivative in b.
__device__ float soft_score(const float h[6], float tau, const float b[3], float *ds, float *db) {
  const float xx = h[0], xy = h[1], xz = h[2], yy = h[3], yz = h[4], zz = h[5];
  const float t2 = tau * tau, t3 = t2 * tau;
  const float m2 = xx * yy - xy * xy;
  const float det = xx * yy * zz + 2.0f * xy * yz * xz - xx * yz * yz - yy * xz * xz - zz * xy * xy;
  const float A = sigm((b[0] - xx) / tau), B = sigm((m2 - b[1]) / t2), C = sigm((b[2] - det) / t3);
  const float s = A * B * C;
  const float ca = -(1.0f - A) / tau, cb = (1.0f - B) / t2, cc = -(1.0f - C) / t3;
  if (ds) {
    // d det / d (xx, xy, xz, yy, yz, zz)
    const float dd[6] = {yy * zz - yz * yz, 2.0f * yz * xz - 2.0f * zz * xy, 2.0f * xy * yz - 2.0f * yy * xz,
                         xx * zz - xz * xz, 2.0f * xy * xz - 2.0f * xx * yz, xx * yy - xy * xy};
    const float dm2[6] = {yy, -2.0f * xy, 0.0f, xx, 0.0f, 0.0f};
    for (int k = 0; k < 6; k++) ds[k] = s * ((k == 0 ? ca : 0.0f) + cb * dm2[k] + cc * dd[k]);
  }
  if (db) {
    db[0] = -s * ca;
    db[1] = -s * cb;
    db[2] = -s * cc;
  }
  return s;
}

// Forward at the points: scores (optional) and the loss (double, out must start at zero).
__global__ void k_soft_points(const float *dog, SoftGeom g, const int32_t *pos, int n_pos, const int32_t *neg,
                              int n_neg, float tau, SoftThresh b, float *scores, double *loss) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pos + n_neg) return;
  const int32_t *q = i < n_pos ? pos + 3 * i : neg + 3 * (i - n_pos);
  const SoftPoint p{q[2], q[1], q[0]};
  float h[6];
  soft_hessian(dog, g, p, h);
  const float s = soft_score(h, tau, b.v, nullptr, nullptr);
  if (scores) scores[i] = s;
  atomicAdd(loss, i < n_pos ? (double)s / n_pos : -(double)s / n_neg);
}

// Backward at the points: d loss / d dog scattered into gdog (which must start at zero), and
// d loss / d thresholds summed into gb[0..2] (double, zeroed first) when gb is given.
__global__ void k_soft_points_adj(const float *dog, SoftGeom g, const int32_t *pos, int n_pos, const int32_t *neg,
                                  int n_neg, float tau, SoftThresh b, float grad_loss, const float *d_grad_loss, double *gdog,
                                  double *gb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_pos + n_neg) return;
  if (d_grad_loss) grad_loss = __ldg(d_grad_loss);
  const int32_t *q = i < n_pos ? pos + 3 * i : neg + 3 * (i - n_pos);
  const SoftPoint p{q[2], q[1], q[0]};
  float h[6], ds[6], db[3];
  soft_hessian(dog, g, p, h);
  soft_score(h, tau, b.v, ds, db);
  const float w = i < n_pos ? grad_loss / (float)n_pos : -grad_loss / (float)n_neg;
  for (int k = 0; k < 6; k++) ds[k] *= w;
  soft_hessian_adj(gdog, g, p, ds);
  if (gb)
    for (int k = 0; k < 3; k++) atomicAdd(gb + k, (double)db[k] * (double)w);
}

__global__ void k_soft_to_float(const double *in, float *out, int n) {
  const int i = threadIdx.x;
  if (i < n) out[i] = (float)in[i];
}

__global__ void k_soft_gdog(const double *in, float *out, int64_t N) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) out[i] = (float)in[i];
}

// ---- the DoG and its derivatives at the points' own neighbourhoods
//
// The loss reads the DoG at 19 positions around each sample point (the Hessian's stencil), and
// d loss / d DoG is zero everywhere else, so with few points the dense Gaussian passes (6
// forward, 16 for the sigma gradients, 6 for the input gradient) compute values that nothing
// reads.  Here a block takes one point at a time: it stages the normalized volume around the
// point (stencil plus the taps' reach) in shared memory, runs the separable passes on the 5 x 5 x 5
// stencil only (x on the lines the y and z taps reach, then y, then z at the 19 positions; both
// scales in one phase), and forms score, derivatives and sums from them.  Every DoG value is the
// dense passes' fold, tap by tap in the same order; a tap outside the volume multiplies a staged
// zero instead of being skipped, which leaves the sum as it is.  The adjoint spreads the stencil's
// gradient through the same taps (z, y, then x) and adds the patch to the normalized volume's
// gradient, one reduction per voxel and point: in float32, or (GT) in doubles where many points may share a voxel.
// What bounds it: the phases' latency (twelve barriers a point) and shared-memory loads; 48 KB and
// 256 threads a block at sigmas 2.0 / 3.2, four blocks per SM.  128x512x512, 4000 points, sigmas
// (2.0, 2.0, 1.5, 3.2, 3.2, 2.4): 98 us forward and 209 us backward, where the 28 dense passes took
// 4.8 ms (the whole forward + backward 10.99 -> 6.23 ms).
constexpr int kSoftPtThreads = 256;
constexpr int kSoftStencil = 19;
constexpr int kSoftPadX = 2 * kSoftMaxRadius + 6;

struct SoftTapSet {
  SoftTaps plain[6], deriv[6];   // x1, y1, z1, x2, y2, z2
};

// Reaches of the staged box (the larger scale's per axis) and the layout of the shared memory.
struct SoftBox {
  int r[3];   // x, y, z
  __host__ __device__ int e(int a) const { return 5 + 2 * r[a]; }
  __host__ __device__ int tile() const { return e(0) * e(1) * e(2); }
  __host__ __device__ int lines() const { return e(1) * e(2); }
  // floats: the tile; per scale two x-pass buffers of 5 outputs per line (the adjoint's y buffers) and
  // three y-pass buffers of 25 columns (the adjoint's z buffers); the plain taps, the x ones padded
  __host__ __device__ int floats() const {
    return tile() + 20 * lines() + 150 * e(2) + 6 * kSoftMaxTaps + 2 * kSoftPadX;
  }
};

// the stencil's position k as offsets from the point (0: the point; 1-6: +-2 along an axis; 7-18: the
// twelve edge neighbours, xy, xz and yz pairs)
__device__ __forceinline__ void soft_stencil(int k, int &dx, int &dy, int &dz) {
  dx = dy = dz = 0;
  if (k == 0) return;
  if (k < 7) {
    const int v = (k & 1) ? 2 : -2, a = (k - 1) >> 1;
    if (a == 0) dx = v;
    else if (a == 1) dy = v;
    else dz = v;
    return;
  }
  const int m = k - 7, pair = m >> 2, u = (m & 1) ? 1 : -1, v = (m & 2) ? 1 : -1;
  if (pair == 0) { dx = u; dy = v; }
  else if (pair == 1) { dx = u; dz = v; }
  else { dy = u; dz = v; }
}
__device__ __forceinline__ int soft_at(int dx, int dy, int dz) { return ((dz + 2) * 5 + dy + 2) * 5 + dx + 2; }

// element e of soft_hessian on the 5 x 5 x 5 cube around p instead of the volume
__device__ __forceinline__ float soft_hessian_cube(const float *f, const SoftGeom &g, SoftPoint p, int e) {
  float v = 0.0f;
  for (int sb = -1; sb <= 1; sb += 2) {
    int qx = 0, qy = 0, qz = 0;
    soft_step(h_outer(e), sb, qx, qy, qz);
    if (!soft_in(g, p.x + qx, p.y + qy, p.z + qz)) continue;
    int ax = qx, ay = qy, az = qz, bx = qx, by = qy, bz = qz;
    soft_step(h_inner(e), 1, ax, ay, az);
    soft_step(h_inner(e), -1, bx, by, bz);
    const float ga = 0.5f * (f[soft_at(ax, ay, az)] - f[soft_at(bx, by, bz)]);
    v += sb > 0 ? ga : -ga;
  }
  return 0.5f * v;
}

// what soft_hessian_adj adds at the stencil's position k: +-gh / 4 of the element whose two steps lead
// there, where the step between them (along the outer axis) stays inside the volume
__device__ __forceinline__ float soft_hessian_coef(const SoftGeom &g, SoftPoint p, int k, const float gh[6]) {
  if (k == 0) {
    const float gd[3] = {gh[0], gh[3], gh[5]};
    float c = 0.0f;
    for (int a = 0; a < 3; a++)
      for (int sb = -1; sb <= 1; sb += 2) {
        int qx = 0, qy = 0, qz = 0;
        soft_step(a, sb, qx, qy, qz);
        if (soft_in(g, p.x + qx, p.y + qy, p.z + qz)) c -= 0.25f * gd[a];
      }
    return c;
  }
  int dx, dy, dz;
  soft_stencil(k, dx, dy, dz);
  if (k < 7) {
    const int a = (k - 1) >> 1;
    return soft_in(g, p.x + dx / 2, p.y + dy / 2, p.z + dz / 2) ? 0.25f * (a == 0 ? gh[0] : a == 1 ? gh[3] : gh[5]) : 0.0f;
  }
  const int pair = (k - 7) >> 2;   // xy: outer y; xz, yz: outer z
  const int qy = pair == 0 ? dy : 0, qz = pair == 0 ? 0 : dz;
  const float s = (float)((dx ? dx : 1) * (dy ? dy : 1) * (dz ? dz : 1));
  return soft_in(g, p.x, p.y + qy, p.z + qz) ? 0.25f * s * (pair == 0 ? gh[1] : pair == 1 ? gh[2] : gh[4]) : 0.0f;
}

// BWD false: scores (optional) and the loss into acc[0].  BWD true: the sums the sigma
// gradients are formed from into acc[0..6] (as soft_backward's dense passes leave them), the
// threshold gradients into gb[0..2], and, when gnorm is given, the gradient of the normalized volume
// added to it.  All sums are doubles that must start at zero.
template <bool BWD, class GT>
__global__ void __launch_bounds__(kSoftPtThreads, 4)
    k_soft_points_local(const float *norm, SoftGeom g, const int32_t *pos, int n_pos, const int32_t *neg, int n_neg,
                        const __grid_constant__ SoftTapSet T, SoftBox box, float nrm, float tau, SoftThresh b,
                        float grad_loss, const float *d_grad_loss, float *scores, double *acc, double *gb, GT *gnorm) {
  extern __shared__ float sm[];
  __shared__ float fv[2][4][kSoftStencil];   // per scale: plain, d/dz, d/dy, d/dx
  __shared__ float cube[125], coef[125];     // DoG and d loss / d DoG around the point (0 off the stencil)
  __shared__ float hs[6], ds[6];
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  if (d_grad_loss) grad_loss = __ldg(d_grad_loss);
  const int ex = box.e(0), ey = box.e(1), ez = box.e(2), L = box.lines();
  float *tile = sm;
  float *xl = tile + box.tile();             // [scale][plain, derivative][lines][5]
  float *yl = xl + 20 * L;                   // [scale][3][25][ez]
  float *tap = yl + 150 * ez;                // [6][kSoftMaxTaps] plain taps: the adjoint's lanes read different ones
  float *padx = tap + 6 * kSoftMaxTaps;      // [2][kSoftPadX] x taps by staged column, zeros around
  for (int i = t; i < 6 * kSoftMaxTaps; i += kSoftPtThreads) tap[i] = T.plain[i / kSoftMaxTaps].k[i % kSoftMaxTaps];
  for (int i = t; i < 2 * kSoftPadX; i += kSoftPtThreads) {
    const SoftTaps &P = T.plain[3 * (i / kSoftPadX)];
    const int j = i % kSoftPadX - (box.r[0] - P.r);
    padx[i] = j >= 0 && j <= 2 * P.r ? P.k[j] : 0.0f;
  }
  for (int i = t; i < 125; i += kSoftPtThreads) cube[i] = coef[i] = 0.0f;
  const int l1y = 5 + 2 * T.plain[1].r, l1z = 5 + 2 * T.plain[2].r, l2y = 5 + 2 * T.plain[4].r, l2z = 5 + 2 * T.plain[5].r;
  const int lines1 = l1y * l1z, lines2 = l2y * l2z, cols1 = 5 * l1z, cols2 = 5 * l2z;
  // this thread's walk over the tile: element t, then 256 further each time
  const int sx = kSoftPtThreads % ex, sl = kSoftPtThreads / ex;
  const int xi0 = t % ex, yi0 = (t / ex) % ey, zi0 = t / (ex * ey);
  int kx, ky, kz;                            // the stencil position of lane % 19's products
  soft_stencil(lane < kSoftStencil ? lane : 0, kx, ky, kz);
  double sum = 0.0;                          // lane 0 of warp w < 7: acc[w]; thread 0 without BWD: the loss
  double gsum[3] = {0.0, 0.0, 0.0};
  const int n = n_pos + n_neg;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    const int32_t *q = i < n_pos ? pos + 3 * (int64_t)i : neg + 3 * (int64_t)(i - n_pos);
    const SoftPoint p{q[2], q[1], q[0]};
    const int x0 = p.x - 2 - box.r[0], y0 = p.y - 2 - box.r[1], z0 = p.z - 2 - box.r[2];
    __syncthreads();   // the previous point is done with the shared memory
    for (int k = t, xi = xi0, yi = yi0, zi = zi0; k < box.tile(); k += kSoftPtThreads) {
      const int x = x0 + xi, y = y0 + yi, z = z0 + zi;
      tile[k] = soft_in(g, x, y, z) ? __ldg(norm + ((int64_t)z * g.H + y) * g.W + x) : 0.0f;
      xi += sx;
      yi += sl;
      if (xi >= ex) { xi -= ex; yi++; }
      while (yi >= ey) { yi -= ey; zi++; }
    }
    __syncthreads();
    // x: five outputs per line, plain taps and (BWD) derivative taps
    for (int m = t; m < lines1 + lines2; m += kSoftPtThreads) {
      const int sc = m >= lines1, l = sc ? m - lines1 : m, ly_n = sc ? l2y : l1y;
      const SoftTaps &px = T.plain[3 * sc];
      const int ly = l % ly_n, lz = l / ly_n, rx = px.r;
      const float *w = tile + ((lz + box.r[2] - T.plain[3 * sc + 2].r) * ey + ly + box.r[1] - T.plain[3 * sc + 1].r) * ex +
                       box.r[0] - rx;
      float a[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, d[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
      float v[5] = {w[0], w[1], w[2], w[3], 0.f};
      for (int j = 0; j <= 2 * rx; j++) {
        v[4] = w[j + 4];
        const float k0 = px.k[j], k1 = BWD ? T.deriv[3 * sc].k[j] : 0.0f;
#pragma unroll
        for (int o = 0; o < 5; o++) {
          a[o] = __fmaf_rn(k0, v[o], a[o]);
          if (BWD) d[o] = __fmaf_rn(k1, v[o], d[o]);
        }
#pragma unroll
        for (int o = 0; o < 4; o++) v[o] = v[o + 1];
      }
      float *out = xl + (2 * sc * L + l) * 5;
#pragma unroll
      for (int o = 0; o < 5; o++) {
        out[o] = a[o];
        if (BWD) out[L * 5 + o] = d[o];
      }
    }
    __syncthreads();
    // y: field 0 plain of plain, 1 derivative of plain, 2 plain of the x derivative
    constexpr int NY = BWD ? 3 : 1, NF = BWD ? 4 : 1;
    for (int m = t; m < NY * (cols1 + cols2); m += kSoftPtThreads) {
      const int sc = m >= NY * cols1, mm = sc ? m - NY * cols1 : m, cols = sc ? cols2 : cols1, ly_n = sc ? l2y : l1y;
      const int f = mm / cols, c = mm % cols, x = c % 5, z = c / 5, ry = T.plain[3 * sc + 1].r;
      const float *w = xl + ((2 * sc + (f == 2)) * L + z * ly_n) * 5 + x;
      const float *kk = f == 1 ? T.deriv[3 * sc + 1].k : T.plain[3 * sc + 1].k;
      float a[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, v[5] = {w[0], w[5], w[10], w[15], 0.f};
      for (int j = 0; j <= 2 * ry; j++) {
        v[4] = w[(j + 4) * 5];
        const float k0 = kk[j];
#pragma unroll
        for (int o = 0; o < 5; o++) a[o] = __fmaf_rn(k0, v[o], a[o]);
#pragma unroll
        for (int o = 0; o < 4; o++) v[o] = v[o + 1];
      }
#pragma unroll
      for (int o = 0; o < 5; o++) yl[((3 * sc + f) * 25 + o * 5 + x) * ez + z] = a[o];
    }
    __syncthreads();
    // z at the stencil: plain, d/dz, d/dy, d/dx
    for (int m = t; m < 2 * NF * kSoftStencil; m += kSoftPtThreads) {
      const int k = m % kSoftStencil, f = (m / kSoftStencil) % NF, sc = m / (kSoftStencil * NF);
      int dx, dy, dz;
      soft_stencil(k, dx, dy, dz);
      const float *w = yl + ((3 * sc + (f < 2 ? 0 : f - 1)) * 25 + (dy + 2) * 5 + dx + 2) * ez + dz + 2;
      const float *kk = f == 1 ? T.deriv[3 * sc + 2].k : T.plain[3 * sc + 2].k;
      const int rz = T.plain[3 * sc + 2].r;
      float a = 0.0f;
      for (int j = 0; j <= 2 * rz; j++) a = __fmaf_rn(kk[j], w[j], a);
      fv[sc][f][k] = a;
    }
    __syncthreads();
    if (warp == 0) {
      const bool in = lane < kSoftStencil && soft_in(g, p.x + kx, p.y + ky, p.z + kz);
      if (lane < kSoftStencil) cube[soft_at(kx, ky, kz)] = in ? nrm * (fv[0][0][lane] - fv[1][0][lane]) : 0.0f;
      __syncwarp();
      if (lane < 6) hs[lane] = soft_hessian_cube(cube, g, p, lane);
      __syncwarp();
      if (lane == 0) {
        float h[6];
        for (int k = 0; k < 6; k++) h[k] = hs[k];
        if (BWD) {
          float dh[6], db[3];
          soft_score(h, tau, b.v, dh, db);
          const float w = i < n_pos ? grad_loss / (float)n_pos : -grad_loss / (float)n_neg;
          for (int k = 0; k < 6; k++) ds[k] = dh[k] * w;
          for (int k = 0; k < 3; k++) gsum[k] += (double)db[k] * (double)w;
        } else {
          const float s = soft_score(h, tau, b.v, nullptr, nullptr);
          if (scores) scores[i] = s;
          sum += i < n_pos ? (double)s / n_pos : -(double)s / n_neg;
        }
      }
      if (BWD) {
        __syncwarp();
        float gh[6];
        for (int k = 0; k < 6; k++) gh[k] = ds[k];
        if (lane < kSoftStencil) coef[soft_at(kx, ky, kz)] = in ? soft_hessian_coef(g, p, lane, gh) : 0.0f;
      }
    }
    if (!BWD) continue;
    __syncthreads();
    if (acc && warp < 7) {
      // <gradient, field> of warp w: w = 3 scale + axis, or the DoG itself
      double v = 0.0;
      if (lane < kSoftStencil && soft_in(g, p.x + kx, p.y + ky, p.z + kz)) {
        const int at = soft_at(kx, ky, kz);
        v = (double)coef[at] * (double)(warp == 6 ? cube[at] : fv[warp / 3][3 - warp % 3][lane]);
      }
      for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
      sum += v;
    }
    if (!gnorm) continue;
    // the transposed passes: z (25 columns), y (5 columns of lines), x into the tile
    for (int m = t; m < 2 * 25 * ez; m += kSoftPtThreads) {
      const int sc = m >= 25 * ez, r = sc ? m - 25 * ez : m, c = r / ez, z = r % ez;
      const int rz = T.plain[3 * sc + 2].r;
      const float *kk = tap + (3 * sc + 2) * kSoftMaxTaps;
      float a = 0.0f;
#pragma unroll
      for (int k = 0; k < 5; k++) {
        const int j = z - (box.r[2] - rz) - k;
        if (j >= 0 && j <= 2 * rz) a = __fmaf_rn(coef[k * 25 + c], kk[j], a);
      }
      yl[m] = a;
    }
    __syncthreads();
    for (int m = t; m < 10 * L; m += kSoftPtThreads) {
      const int xs = m / L, l = m % L, sc = xs >= 5, x = sc ? xs - 5 : xs;   // xs = 5 scale + column
      const int y = l % ey, z = l / ey, ry = T.plain[3 * sc + 1].r, off = box.r[1] - ry;
      const float *kk = tap + (3 * sc + 1) * kSoftMaxTaps;
      const float *w = yl + (sc * 25 + x) * ez + z;
      float a = 0.0f;
#pragma unroll
      for (int k = 0; k < 5; k++) {
        const int j = y - off - k;
        if (j >= 0 && j <= 2 * ry) a = __fmaf_rn(w[k * 5 * ez], kk[j], a);
      }
      xl[m] = a;
    }
    __syncthreads();
    for (int l = t; l < L; l += kSoftPtThreads) {
      float c1[5], c2[5], t1[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, t2[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int o = 0; o < 5; o++) {
        c1[o] = xl[o * L + l];
        c2[o] = xl[(5 + o) * L + l];
      }
      for (int xi = 0; xi < ex; xi++) {
#pragma unroll
        for (int o = 4; o > 0; o--) { t1[o] = t1[o - 1]; t2[o] = t2[o - 1]; }
        t1[0] = padx[xi];
        t2[0] = padx[kSoftPadX + xi];
        float a = 0.0f, c = 0.0f;
#pragma unroll
        for (int o = 0; o < 5; o++) {
          a = __fmaf_rn(c1[o], t1[o], a);
          c = __fmaf_rn(c2[o], t2[o], c);
        }
        tile[l * ex + xi] = nrm * (a - c);
      }
    }
    __syncthreads();
    for (int k = t, xi = xi0, yi = yi0, zi = zi0; k < box.tile(); k += kSoftPtThreads) {
      const int x = x0 + xi, y = y0 + yi, z = z0 + zi;
      const float v = tile[k];
      if (v != 0.0f && soft_in(g, x, y, z)) atomicAdd(gnorm + ((int64_t)z * g.H + y) * g.W + x, (GT)v);
      xi += sx;
      yi += sl;
      if (xi >= ex) { xi -= ex; yi++; }
      while (yi >= ey) { yi -= ey; zi++; }
    }
  }
  if (!BWD) {
    if (t == 0) atomicAdd(acc, sum);
    return;
  }
  if (acc && warp < 7 && lane == 0) atomicAdd(acc + warp, sum);
  if (gb && t == 0)
    for (int k = 0; k < 3; k++) atomicAdd(gb + k, gsum[k]);
}

// d loss / d sigma from the sums <gradient, derivative fields> (h[0..5]) and <gradient, DoG>
// (h[6]): the normalizer times the field's sum, plus the normalizer's own derivative
// gamma normalizer / sigma.  A normalized volume with a value that is not finite (*bad) makes every
// dense field, and so every sum, NaN; sums taken at the points alone say so here.
struct SoftSigma {
  float v[6];
};
__global__ void k_soft_sigma_grad(const double *h, const unsigned *bad, SoftSigma s, float nrm, float gamma, float *out) {
  const int k = threadIdx.x;
  if (k >= 6) return;
  double v = (double)(k < 3 ? nrm : -nrm) * h[k];
  if (k < 3) v = __dadd_rn(v, __dmul_rn((double)gamma / s.v[k], h[6]));
  out[k] = bad && *bad ? __int_as_float(0x7FC00000) : (float)v;
}

// ------------------------------------------------------------------ host side
namespace {

struct SoftRun {
  const hdog_soft_params &p;
  SoftGeom g;
  int64_t N;
  cudaStream_t st;
  float *w;      // workspace slots of slot_floats(N) floats (after the accumulators)
  double *acc;   // 16 doubles at the start of the workspace: sums [0, 14), then the flags
  // set by the forward chain: [0] a normalized value is not finite, [1] the DoG slot is filled
  unsigned *flags() const { return reinterpret_cast<unsigned *>(acc + 14); }
  unsigned blocks() const { return ceil_div(N, 256); }
  static int64_t slot_floats(int64_t n) { return (n + 31) / 32 * 32; }   // whole 128-byte lines
  float *slot(int k) const { return w + k * slot_floats(N); }
  float2 *pair(int k) const { return reinterpret_cast<float2 *>(slot(k)); }   // slots k and k + 1
};

// Kept for the backward: the extremes after the x and the y pass, the box means (pairs, min and max
// side in one float2), the normalized volume, the DoG; scratch: two pairs and one volume.  The dense
// Gaussian passes use the pairs' halves.
enum { S_MM1 = 0, S_MM2 = 2, S_ED = 4, S_NORM = 6, S_DOG = 7, S_PA = 8, S_PB = 10, S_GB = 12, kSoftSlots = 13,
       S_T1 = S_PA, S_T2 = S_PA + 1, S_T3 = S_PB, S_GDOG = S_PB + 1 };

// Normalized Gaussian taps of sigma (or their derivative in sigma), radius (int)(2 sigma + 0.5).
SoftTaps gauss_taps_f(double sigma, bool derivative) {
  SoftTaps t;
  memset(&t, 0, sizeof(t));
  const int r = (int)(2.0 * sigma + 0.5);
  t.r = r;
  double e[kSoftMaxTaps], sum = 0.0, m2 = 0.0;
  for (int k = -r; k <= r; k++) {
    e[k + r] = exp(-0.5 * k * k / (sigma * sigma));
    sum += e[k + r];
  }
  for (int k = -r; k <= r; k++) m2 += e[k + r] / sum * (double)k * k;
  for (int k = -r; k <= r; k++) {
    const double tk = e[k + r] / sum;
    t.k[k + r] = (float)(derivative ? tk * ((double)k * k - m2) / (sigma * sigma * sigma) : tk);
  }
  return t;
}

void pass(const SoftRun &R, const float *in, float *out, int axis, const SoftTaps &T, const unsigned *skip = nullptr) {
  const SoftGeom &g = R.g;
  if (axis == 0) {
    const unsigned blocks = (unsigned)(ceil_div(g.W, kSoftTileX) * ceil_div((int64_t)g.H * g.D, kSoftRowsX));
    KLAUNCH("k_soft_pass_x", R.st, (k_soft_pass_x<<<blocks, kSoftTileX, 0, R.st>>>(in, out, g, T, skip)));
    return;
  }
  const size_t smem = (size_t)(kSoftTileYZ + 2 * T.r) * 32 * sizeof(float);
  const int n = axis == 1 ? g.H : g.D, other = axis == 1 ? g.D : g.H;
  const dim3 grid((unsigned)ceil_div(g.W, 32), (unsigned)ceil_div(n, kSoftTileYZ), (unsigned)other);
  if (axis == 1)
    KLAUNCH("k_soft_pass_y", R.st, (k_soft_pass_yz<1><<<grid, dim3(32, 8), smem, R.st>>>(in, out, g, T, skip)));
  else
    KLAUNCH("k_soft_pass_z", R.st, (k_soft_pass_yz<2><<<grid, dim3(32, 8), smem, R.st>>>(in, out, g, T, skip)));
}

// the correlation along z with T, summed against w into *acc (double) instead of stored
void pass_z_dot(const SoftRun &R, const float *in, const SoftTaps &T, const float *w, double *acc) {
  const SoftGeom &g = R.g;
  const size_t smem = (size_t)(kSoftTileYZ + 2 * T.r) * 32 * sizeof(float);
  const dim3 grid((unsigned)ceil_div(g.W, 32), (unsigned)ceil_div(g.D, kSoftTileYZ), (unsigned)g.H);
  KLAUNCH("k_soft_pass_z_dot", R.st, (k_soft_pass_yz<2, kEpiDot><<<grid, dim3(32, 8), smem, R.st>>>(
                                         in, nullptr, g, T, nullptr, w, acc)));
}

// the separable Gaussian (x, y, then z) with the DoG difference folded into the z pass:
// out = scale * (sub - in * G), the same operations as a separate difference kernel
void conv3_diff(const SoftRun &R, const float *in, float *out, const SoftTaps &tx, const SoftTaps &ty,
                const SoftTaps &tz, float *t1, float *t2, const float *sub, float scale, const unsigned *skip) {
  pass(R, in, t1, 0, tx, skip);
  pass(R, t1, t2, 1, ty, skip);
  const SoftGeom &g = R.g;
  const size_t smem = (size_t)(kSoftTileYZ + 2 * tz.r) * 32 * sizeof(float);
  const dim3 grid((unsigned)ceil_div(g.W, 32), (unsigned)ceil_div(g.D, kSoftTileYZ), (unsigned)g.H);
  KLAUNCH("k_soft_pass_z_diff", R.st, (k_soft_pass_yz<2, kEpiDiff><<<grid, dim3(32, 8), smem, R.st>>>(
                                          t2, out, g, tz, skip, sub, nullptr, scale)));
}

// ---- the normalization's windows
constexpr size_t kSoftMaxSmem = 220 * 1024;
constexpr int kSoftColWarps[3] = {0, 8, 4};   // warps of the column passes along y and z

// The allowance belongs to the kernel, not to the launch, so it is the largest of any call: a smaller one could take
// away what another host thread has just asked for.
template <class F>
void allow_smem(F *fn, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSoftMaxSmem);
}

// Grid of a column pass: 32 columns x the other coordinate x segments of the line, which is cut while the
// columns alone are fewer than `blocks` blocks, into segments of at least `shortest`.
dim3 col_grid(const SoftGeom &g, int axis, int shortest, int64_t blocks, int &seg) {
  const int n = axis == 1 ? g.H : g.D, other = axis == 1 ? g.D : g.H;
  const int64_t cols = (int64_t)ceil_div(g.W, 32) * other;
  const int64_t want = std::max<int64_t>(1, (blocks + cols - 1) / cols);
  seg = std::min<int64_t>(n, std::max<int64_t>(ceil_div(n, want), shortest));
  return dim3((unsigned)ceil_div(g.W, 32), (unsigned)other, (unsigned)ceil_div(n, seg));
}

dim3 short_grid(const SoftGeom &g, int axis) {
  const int n = axis == 1 ? g.H : g.D, other = axis == 1 ? g.D : g.H;
  return dim3((unsigned)ceil_div(g.W, 32), (unsigned)other, (unsigned)ceil_div(n, 8 * kSoftShort));
}

// Extremes along `axis`: the volume itself (axis 0) or a pair in, a pair out.
void ext_pass(const SoftRun &R, const void *in, float2 *out, int axis, int r) {
  const SoftGeom &g = R.g;
  const float2 *in2 = static_cast<const float2 *>(in);
  if (axis == 0) {
    const float *v = static_cast<const float *>(in);
    const int64_t rows = (int64_t)g.H * g.D;
    if (r >= 4 && r <= 255) {
      switch ((8 - 2 * r % 8) % 8 + (row_of_8(r, g.W, rows, INT_MAX) ? 1 : 0)) {
#define HDOG_CASE(Q)                                                                                                  \
  case Q:                                                                                                             \
    KLAUNCH("k_soft_ext_rows", R.st, (k_soft_ext_rows<32, Q><<<ceil_div(rows, kSoftRowWarps), 32 * kSoftRowWarps, 0,  \
                                                               R.st>>>(v, out, g, r)));                               \
    return;                                                                                                           \
  case Q + 1:                                                                                                         \
    KLAUNCH("k_soft_ext_rows", R.st, (k_soft_ext_rows<8, Q><<<ceil_div(rows, 4 * kSoftRowWarps), 32 * kSoftRowWarps,  \
                                                              0, R.st>>>(v, out, g, r)));                             \
    return;
        HDOG_CASE(0) HDOG_CASE(2) HDOG_CASE(4) HDOG_CASE(6)
#undef HDOG_CASE
      }
    }
    KLAUNCH("k_soft_ext_far", R.st, (k_soft_ext_far<true><<<R.blocks(), 256, 0, R.st>>>(in, out, g, axis, r, R.N)));
    return;
  }
  if (r < 4) {
    const dim3 grid = short_grid(g, axis), block(32, 8);
#define HDOG_CASE(A, Q) \
  if (axis == A && r == Q) KLAUNCH("k_soft_ext_short", R.st, (k_soft_ext_short<A, Q><<<grid, block, 0, R.st>>>(in2, out, g)));
    HDOG_CASE(1, 0) HDOG_CASE(1, 1) HDOG_CASE(1, 2) HDOG_CASE(1, 3) HDOG_CASE(2, 0) HDOG_CASE(2, 1) HDOG_CASE(2, 2) HDOG_CASE(2, 3)
#undef HDOG_CASE
    return;
  }
  const int nw = kSoftColWarps[axis];
  const size_t smem = (size_t)ext_cols_rows(r, kSoftB, nw) * 32 * sizeof(float2);
  if (smem > kSoftMaxSmem) {
    KLAUNCH("k_soft_ext_far", R.st, (k_soft_ext_far<false><<<R.blocks(), 256, 0, R.st>>>(in, out, g, axis, r, R.N)));
    return;
  }
  int seg;
  const dim3 grid = col_grid(g, axis, std::max(nw * kSoftB, 2 * r), 152 * 8, seg);
  if (axis == 1) {
    allow_smem(k_soft_ext_cols<1, kSoftColWarps[1]>, smem);
    KLAUNCH("k_soft_ext_y", R.st, (k_soft_ext_cols<1, kSoftColWarps[1]><<<grid, dim3(32, nw), smem, R.st>>>(in2, out, g, r, seg)));
  } else {
    allow_smem(k_soft_ext_cols<2, kSoftColWarps[2]>, smem);
    KLAUNCH("k_soft_ext_z", R.st, (k_soft_ext_cols<2, kSoftColWarps[2]><<<grid, dim3(32, nw), smem, R.st>>>(in2, out, g, r, seg)));
  }
}

// The adjoint of ext_pass: the gradient pair gout, through the pass's input src, added to gin (axis 0: the
// volume's gradient; else a zeroed pair).
void ext_adj(const SoftRun &R, const void *src, const float2 *gout, float *gin, int axis, int r) {
  const SoftGeom &g = R.g;
  if (axis == 0) {
    const float *v = static_cast<const float *>(src);
    const int64_t rows = (int64_t)g.H * g.D;
    if (r >= 4 && r <= 255) {
      switch ((8 - 2 * r % 8) % 8 + (row_of_8(r, g.W, rows, INT_MAX) ? 1 : 0)) {
#define HDOG_CASE(Q)                                                                                                      \
  case Q:                                                                                                                 \
    KLAUNCH("k_soft_ext_adj_rows", R.st, (k_soft_ext_adj_rows<32, Q><<<ceil_div(rows, kSoftRowWarps), 32 * kSoftRowWarps, \
                                                                       0, R.st>>>(v, gout, gin, g, r)));                  \
    return;                                                                                                               \
  case Q + 1:                                                                                                             \
    KLAUNCH("k_soft_ext_adj_rows", R.st, (k_soft_ext_adj_rows<8, Q><<<ceil_div(rows, 4 * kSoftRowWarps),                  \
                                                                      32 * kSoftRowWarps, 0, R.st>>>(v, gout, gin, g, r))); \
    return;
        HDOG_CASE(0) HDOG_CASE(2) HDOG_CASE(4) HDOG_CASE(6)
#undef HDOG_CASE
      }
    }
    KLAUNCH("k_soft_ext_adj_far", R.st, (k_soft_ext_adj_far<true><<<R.blocks(), 256, 0, R.st>>>(src, gout, gin, g, axis, r, R.N)));
    return;
  }
  if (r < 4) {
    const dim3 grid = short_grid(g, axis), block(32, 8);
#define HDOG_CASE(A, Q)                                                                                               \
  if (axis == A && r == Q)                                                                                            \
    KLAUNCH("k_soft_ext_adj_short", R.st, (k_soft_ext_adj_short<A, Q><<<grid, block, 0, R.st>>>(                      \
                                              static_cast<const float2 *>(src), gout, reinterpret_cast<float2 *>(gin), g)));
    HDOG_CASE(1, 0) HDOG_CASE(1, 1) HDOG_CASE(1, 2) HDOG_CASE(1, 3) HDOG_CASE(2, 0) HDOG_CASE(2, 1) HDOG_CASE(2, 2) HDOG_CASE(2, 3)
#undef HDOG_CASE
    return;
  }
  const size_t smem = (size_t)ext_cols_rows(r, kSoftB, 1) * 32 * (sizeof(float2) + sizeof(uint16_t));
  if (smem > kSoftMaxSmem) {
    KLAUNCH("k_soft_ext_adj_far", R.st, (k_soft_ext_adj_far<false><<<R.blocks(), 256, 0, R.st>>>(src, gout, gin, g, axis, r, R.N)));
    return;
  }
  int seg;
  const dim3 grid = col_grid(g, axis, std::max(16, r), 152 * 16, seg);   // 16 warps per SM
  const float2 *s2 = static_cast<const float2 *>(src);
  float2 *g2 = reinterpret_cast<float2 *>(gin);
  if (axis == 1) {
    allow_smem(k_soft_ext_adj_cols<1>, smem);
    KLAUNCH("k_soft_ext_adj_y", R.st, (k_soft_ext_adj_cols<1><<<grid, 32, smem, R.st>>>(s2, gout, g2, g, r, seg)));
  } else {
    allow_smem(k_soft_ext_adj_cols<2>, smem);
    KLAUNCH("k_soft_ext_adj_z", R.st, (k_soft_ext_adj_cols<2><<<grid, 32, smem, R.st>>>(s2, gout, g2, g, r, seg)));
  }
}

// Box means of a pair along `axis`, or (ADJ) the transpose; vol given (axis 2): also the normalized volume.
template <bool ADJ>
void box_pass(const SoftRun &R, const float2 *in, float2 *out, int axis, int r, const float *vol = nullptr) {
  const SoftGeom &g = R.g;
  const size_t smem = (size_t)32 * ((kSoftBoxX + 2 * r) | 1) * sizeof(float2);
  if (smem > kSoftMaxSmem) {   // reaches from 376
    KLAUNCH("k_soft_box_far", R.st, (k_soft_box_far<ADJ><<<R.blocks(), 256, 0, R.st>>>(in, out, g, axis, r, R.N)));
    if (vol)
      KLAUNCH("k_soft_norm", R.st, (k_soft_norm<<<R.blocks(), 256, 0, R.st>>>(vol, out, R.slot(S_NORM), R.p.min_intensity, R.N,
                                                                             R.flags())));
    return;
  }
  if (axis == 0) {
    allow_smem(k_soft_box_x<ADJ>, smem);
    const unsigned blocks = (unsigned)(ceil_div(g.W, kSoftBoxX) * ceil_div((int64_t)g.H * g.D, 32));
    KLAUNCH(ADJ ? "k_soft_box_adj_x" : "k_soft_box_x", R.st, (k_soft_box_x<ADJ><<<blocks, 256, smem, R.st>>>(in, out, g, r)));
    return;
  }
  if (axis == 1) {
    constexpr int K = 16;
    const dim3 grid((unsigned)ceil_div(g.W, 32), (unsigned)g.D, (unsigned)ceil_div(g.H, 4 * K));
    KLAUNCH(ADJ ? "k_soft_box_adj_y" : "k_soft_box_y", R.st,
            (k_soft_box_cols<1, K, ADJ, false, 0><<<grid, dim3(32, 4), 0, R.st>>>(in, out, g, r, nullptr, nullptr, 0.0f, nullptr)));
    return;
  }
  constexpr int K = 8;
  const dim3 grid((unsigned)ceil_div(g.W, 32), (unsigned)g.H, (unsigned)ceil_div(g.D, 4 * K));
  switch (r) {
#define HDOG_CASE(RT)                                                                                                   \
  case RT:                                                                                                              \
    if (vol)                                                                                                            \
      KLAUNCH("k_soft_box_z_norm", R.st, (k_soft_box_cols<2, K, false, true, RT><<<grid, dim3(32, 4), 0, R.st>>>(       \
                                             in, out, g, r, vol, R.slot(S_NORM), R.p.min_intensity, R.flags())));       \
    else                                                                                                                \
      KLAUNCH("k_soft_box_adj_z", R.st, (k_soft_box_cols<2, K, true, false, RT><<<grid, dim3(32, 4), 0, R.st>>>(        \
                                            in, out, g, r, nullptr, nullptr, 0.0f, nullptr)));                          \
    return;
    HDOG_CASE(1) HDOG_CASE(2) HDOG_CASE(3) HDOG_CASE(4) HDOG_CASE(5) HDOG_CASE(6) HDOG_CASE(7) HDOG_CASE(8)
#undef HDOG_CASE
  }
  if (vol)
    KLAUNCH("k_soft_box_z_norm", R.st, (k_soft_box_cols<2, K, false, true, 0><<<grid, dim3(32, 4), 0, R.st>>>(
                                           in, out, g, r, vol, R.slot(S_NORM), R.p.min_intensity, R.flags())));
  else
    KLAUNCH("k_soft_box_adj_z", R.st, (k_soft_box_cols<2, K, true, false, 0><<<grid, dim3(32, 4), 0, R.st>>>(
                                          in, out, g, r, nullptr, nullptr, 0.0f, nullptr)));
}

// conv of `in` with taps (tx, ty, tz) along x, y, z -> out (t1, t2 as temporaries)
void conv3(const SoftRun &R, const float *in, float *out, const SoftTaps &tx, const SoftTaps &ty, const SoftTaps &tz,
           float *t1, float *t2, const unsigned *skip = nullptr) {
  pass(R, in, t1, 0, tx, skip);
  pass(R, t1, t2, 1, ty, skip);
  pass(R, t2, out, 2, tz, skip);
}

// The DoG slot from the normalized one (temporaries T1-T3); skip: a device flag that says it is filled.
void dense_dog(const SoftRun &R, const unsigned *skip) {
  const float *s = R.p.sigma;
  const float nrm = (float)pow((double)s[0] * s[1] * s[2], (double)R.p.gamma);
  conv3(R, R.slot(S_NORM), R.slot(S_T3), gauss_taps_f(s[0], false), gauss_taps_f(s[1], false), gauss_taps_f(s[2], false),
        R.slot(S_T1), R.slot(S_T2), skip);
  conv3_diff(R, R.slot(S_NORM), R.slot(S_DOG), gauss_taps_f(s[3], false), gauss_taps_f(s[4], false),
             gauss_taps_f(s[5], false), R.slot(S_T1), R.slot(S_T2), R.slot(S_T3), nrm, skip);
}

// The forward chain into the workspace: min/max chains, box means, norm, and the DoG when the
// score is to be read from the volume.
void forward_chain(const SoftRun &R, const float *vol, bool want_dog) {
  cudaMemsetAsync(R.acc, 0, 16 * sizeof(double), R.st);
  const int rxy = R.p.radius_norm_xy, rz = R.p.radius_norm_z;
  float2 *mm1 = R.pair(S_MM1), *mm2 = R.pair(S_MM2), *pa = R.pair(S_PA), *pb = R.pair(S_PB);
  ext_pass(R, vol, mm1, 0, rxy);
  ext_pass(R, mm1, mm2, 1, rxy);
  ext_pass(R, mm2, pa, 2, rz);
  box_pass<false>(R, pa, pb, 0, rxy);
  box_pass<false>(R, pb, pa, 1, rxy);
  box_pass<false>(R, pa, R.pair(S_ED), 2, rz, vol);
  if (want_dog) {
    dense_dog(R, nullptr);
    cudaMemsetAsync(R.flags() + 1, 1, sizeof(unsigned), R.st);
  }
}

// Whether the DoG is evaluated at the points' neighbourhoods (k_soft_points_local) instead of
// over the volume: when a block's box fits twice on an SM, and the points cost less than the 28 dense
// passes.  Measured (forward + backward, ns): a point 34, 57 and 185 at patches of 1859, 4335 and
// 14297 voxels, so about 20 + 0.011 per voxel; the dense passes 0.16 per voxel of the volume plus about
// 150 us of launches (665-830 us at 64x256x256, 200 us at 32x80x96).  At 64x256x256 that puts the
// line at 12 k points for the middle patch: 8 k took 1.60 against 1.95 ms, 32 k 3.00 against 2.09.
constexpr size_t kSoftLocalSmem = 110 * 1024;

bool points_local(const SoftRun &R, int64_t n, SoftBox &box) {
  for (int a = 0; a < 3; a++)
    box.r[a] = std::max((int)(2.0 * R.p.sigma[a] + 0.5), (int)(2.0 * R.p.sigma[a + 3] + 0.5));
  if ((size_t)box.floats() * sizeof(float) > kSoftLocalSmem) return false;
  return (double)n * (20.0 + 0.011 * box.tile()) <= 0.16 * (double)R.N + 150e3;
}

// Points from which the gradient of the normalized volume is summed in doubles: a float32 sum of n like terms is off by up
// to n / 2^25 of itself (60 k points at one place: 4e-4).  Doubles take 50 of 2490 us more at 512x512x128.
constexpr int64_t kSoftManyPoints = 4096;

template <bool BWD, class GT = float>
void points_launch(const SoftRun &R, const SoftBox &box, const int32_t *pos, int n_pos, const int32_t *neg, int n_neg,
                   float grad_loss, const float *d_grad_loss, float *scores, double *acc, double *gb, GT *gnorm) {
  const hdog_soft_params &p = R.p;
  const int64_t n = (int64_t)n_pos + n_neg;
  if (n == 0) return;
  SoftTapSet T;
  for (int k = 0; k < 6; k++) {
    T.plain[k] = gauss_taps_f(p.sigma[k], false);
    T.deriv[k] = gauss_taps_f(p.sigma[k], true);
  }
  SoftThresh b;
  for (int k = 0; k < 3; k++) b.v[k] = p.thresh[k];
  const float *s = p.sigma;
  const float nrm = (float)pow((double)s[0] * s[1] * s[2], (double)p.gamma);
  const size_t smem = (size_t)box.floats() * sizeof(float);
  if (smem > 44 * 1024)   // 48 KB without it, static shared memory included
    cudaFuncSetAttribute(k_soft_points_local<BWD, GT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSoftLocalSmem);
  const unsigned grid = (unsigned)std::min<int64_t>(n, 152 * 8);
  KLAUNCH(BWD ? "k_soft_points_local_adj" : "k_soft_points_local", R.st,
          (k_soft_points_local<BWD, GT><<<grid, kSoftPtThreads, smem, R.st>>>(R.slot(S_NORM), R.g, pos, n_pos, neg, n_neg, T,
                                                                          box, nrm, p.tau, b, grad_loss, d_grad_loss, scores,
                                                                          acc, gb, gnorm)));
}

SoftThresh thresh_of(const hdog_soft_params &p) {
  SoftThresh b;
  for (int k = 0; k < 3; k++) b.v[k] = p.thresh[k];
  return b;
}

int check_params(const hdog_soft_params *p, const float *vol, const int32_t *pos, int n_pos, const int32_t *neg,
                 int n_neg, void *work) {
  if (!p || !vol || !work || n_pos < 0 || n_neg < 0 || (n_pos && !pos) || (n_neg && !neg))
    return HDOG_ERR_ARG;
  if (p->width < 1 || p->height < 1 || p->depth < 1 || p->radius_norm_xy < 0 || p->radius_norm_z < 0 ||
      p->radius_norm_xy > 1000 || p->radius_norm_z > 1000 || !(p->tau > 0.0f))
    return HDOG_ERR_PARAM;
  for (int k = 0; k < 6; k++)
    if (!(p->sigma[k] > 0.0f) || (int)(2.0 * p->sigma[k] + 0.5) > kSoftMaxRadius) return HDOG_ERR_SHAPE;
  return HDOG_OK;
}

}  // namespace

size_t soft_workspace_bytes(const hdog_soft_params &p) {
  return 16 * sizeof(double) + (size_t)kSoftSlots * SoftRun::slot_floats((int64_t)p.width * p.height * p.depth) * sizeof(float);
}

int soft_forward(const hdog_soft_params *p, const float *vol, const int32_t *pos, int n_pos, const int32_t *neg,
                 int n_neg, float *loss, float *scores, void *work, cudaStream_t st) {
  const int rc = check_params(p, vol, pos, n_pos, neg, n_neg, work);
  if (rc != HDOG_OK || !loss) return rc != HDOG_OK ? rc : HDOG_ERR_ARG;
  SoftRun R{*p, SoftGeom{p->width, p->height, p->depth}, (int64_t)p->width * p->height * p->depth, st,
            static_cast<float *>(work), nullptr};
  R.acc = static_cast<double *>(work);
  R.w = reinterpret_cast<float *>(R.acc + 16);
  SoftBox box;
  const bool local = points_local(R, (int64_t)n_pos + n_neg, box);
  forward_chain(R, vol, !local);
  if (local)
    points_launch<false>(R, box, pos, n_pos, neg, n_neg, 0.0f, nullptr, scores, R.acc, nullptr, static_cast<float *>(nullptr));
  else if (n_pos + n_neg > 0)
    KLAUNCH("k_soft_points", st, (k_soft_points<<<ceil_div(n_pos + n_neg, 128), 128, 0, st>>>(
                                     R.slot(S_DOG), R.g, pos, n_pos, neg, n_neg, p->tau, thresh_of(*p), scores,
                                     R.acc)));
  k_soft_to_float<<<1, 32, 0, st>>>(R.acc, loss, 1);
  return HDOG_OK;
}

int soft_backward(const hdog_soft_params *p, const float *vol, const int32_t *pos, int n_pos, const int32_t *neg,
                  int n_neg, float grad_loss, float *grad_vol, float *grad_sigma, float *grad_thresh, void *work,
                  cudaStream_t st, bool forward_kept, const float *d_grad_loss) {
  const int rc = check_params(p, vol, pos, n_pos, neg, n_neg, work);
  if (rc != HDOG_OK) return rc;
  SoftRun R{*p, SoftGeom{p->width, p->height, p->depth}, (int64_t)p->width * p->height * p->depth, st,
            static_cast<float *>(work), nullptr};
  R.acc = static_cast<double *>(work);
  R.w = reinterpret_cast<float *>(R.acc + 16);
  const unsigned nb = R.blocks();
  // The backward reads the forward chain's slots (S_MM1 .. S_DOG) and writes only the others,
  // so a workspace that soft_forward filled for the same inputs still holds them.
  SoftBox box;
  const bool local = points_local(R, (int64_t)n_pos + n_neg, box);
  if (!forward_kept) forward_chain(R, vol, !local);
  const float *s = p->sigma;
  const float nrm = (float)pow((double)s[0] * s[1] * s[2], (double)p->gamma);
  // acc[0..5]: <gdog, d dog / d sigma_k> without the normalizer term; acc[6]: <gdog, dog>
  double *gb = R.acc + 8;   // threshold gradients
  cudaMemsetAsync(R.acc, 0, 14 * sizeof(double), st);
  float *gdog = R.slot(S_GDOG);
  const bool many = local && (int64_t)n_pos + n_neg > kSoftManyPoints;
  if (local) {
    double *sums = grad_sigma ? R.acc : nullptr, *thr = grad_thresh ? gb : nullptr;
    if (many) {
      double *gnorm = grad_vol ? reinterpret_cast<double *>(R.slot(S_PA)) : nullptr;   // a pair's two slots
      if (gnorm) cudaMemsetAsync(gnorm, 0, R.N * sizeof(double), st);
      points_launch<true>(R, box, pos, n_pos, neg, n_neg, grad_loss, d_grad_loss, nullptr, sums, thr, gnorm);
    } else {
      float *gnorm = grad_vol ? R.slot(S_GB) : nullptr;
      if (gnorm) cudaMemsetAsync(gnorm, 0, R.N * sizeof(float), st);
      points_launch<true>(R, box, pos, n_pos, neg, n_neg, grad_loss, d_grad_loss, nullptr, sums, thr, gnorm);
    }
  } else {
    // a forward call with fewer points may have left the DoG slot empty
    if (forward_kept) dense_dog(R, R.flags() + 1);
    double *gsum = reinterpret_cast<double *>(R.slot(S_PA));   // a pair's two slots
    cudaMemsetAsync(gsum, 0, R.N * sizeof(double), st);
    if (n_pos + n_neg > 0)
      KLAUNCH("k_soft_points_adj", st, (k_soft_points_adj<<<ceil_div(n_pos + n_neg, 128), 128, 0, st>>>(
                                           R.slot(S_DOG), R.g, pos, n_pos, neg, n_neg, p->tau, thresh_of(*p), grad_loss,
                                           d_grad_loss, gsum, gb)));
    KLAUNCH("k_soft_gdog", st, (k_soft_gdog<<<nb, 256, 0, st>>>(gsum, gdog, R.N)));
  }
  if (grad_thresh) k_soft_to_float<<<1, 32, 0, st>>>(gb, grad_thresh, 3);
  if (grad_sigma) {
    if (!local) {
      const unsigned db = 152 * 4;
      // Per scale: <gdog, C_z C_y C_x norm> with the derivative taps on one axis.  The plain x
      // pass serves the y and z derivatives, and every z pass folds straight into the dot.
      float *nm = R.slot(S_NORM), *t1 = R.slot(S_T1), *t2 = R.slot(S_T2);
      for (int sc = 0; sc < 2; sc++) {
        SoftTaps pl[3], dv[3];
        for (int a = 0; a < 3; a++) {
          pl[a] = gauss_taps_f(s[3 * sc + a], false);
          dv[a] = gauss_taps_f(s[3 * sc + a], true);
        }
        double *acc = R.acc + 3 * sc;
        pass(R, nm, t1, 0, pl[0]);
        pass(R, t1, t2, 1, pl[1]);
        pass_z_dot(R, t2, dv[2], gdog, acc + 2);
        pass(R, t1, t2, 1, dv[1]);
        pass_z_dot(R, t2, pl[2], gdog, acc + 1);
        pass(R, nm, t1, 0, dv[0]);
        pass(R, t1, t2, 1, pl[1]);
        pass_z_dot(R, t2, pl[2], gdog, acc + 0);
      }
      KLAUNCH("k_soft_dot", st, (k_soft_dot<<<db, 256, 0, st>>>(gdog, R.slot(S_DOG), R.N, R.acc + 6)));
    }
    SoftSigma sg;
    for (int k = 0; k < 6; k++) sg.v[k] = s[k];
    KLAUNCH("k_soft_sigma_grad", st, (k_soft_sigma_grad<<<1, 32, 0, st>>>(R.acc, local ? R.flags() : nullptr, sg, nrm,
                                                                         p->gamma, grad_sigma)));
  }
  if (grad_vol) {
    if (!local) {
      // g_norm = normalizer (G1 - G2)^T gdog = normalizer (G1 gdog - G2 gdog)
      conv3(R, gdog, R.slot(S_T3), gauss_taps_f(s[0], false), gauss_taps_f(s[1], false), gauss_taps_f(s[2], false),
            R.slot(S_T1), R.slot(S_T2));
      conv3_diff(R, gdog, R.slot(S_GB), gauss_taps_f(s[3], false), gauss_taps_f(s[4], false), gauss_taps_f(s[5], false),
                 R.slot(S_T1), R.slot(S_T2), R.slot(S_T3), nrm, nullptr);
    }
    // quotient rule: direct term into grad_vol, the box means' gradients into a pair
    float2 *cur = R.pair(S_PA), *next = R.pair(S_PB);
    const auto on16 = [](const void *q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    const bool by4 = on16(vol) && on16(grad_vol) && on16(work);
    const unsigned blocks = by4 ? ceil_div(R.N, 1024) : nb;
    if (many)
      KLAUNCH("k_soft_norm_adj", st, ((by4 ? k_soft_norm_adj<4, double> : k_soft_norm_adj<1, double>)<<<blocks, 256, 0, st>>>(
                                         vol, R.pair(S_ED), reinterpret_cast<const double *>(cur), grad_vol, cur,
                                         p->min_intensity, R.N)));
    else
      KLAUNCH("k_soft_norm_adj", st, ((by4 ? k_soft_norm_adj<4, float> : k_soft_norm_adj<1, float>)<<<blocks, 256, 0, st>>>(
                                         vol, R.pair(S_ED), R.slot(S_GB), grad_vol, cur, p->min_intensity, R.N)));
    // box means transposed z -> y -> x, then the extremes z -> y -> x, each adding to a zeroed pair but the
    // last, which adds straight to the input gradient (holding the quotient rule's direct term)
    const int rr[3] = {p->radius_norm_xy, p->radius_norm_xy, p->radius_norm_z};
    for (int a = 2; a >= 0; a--) {
      if (rr[a] == 0) continue;
      box_pass<true>(R, cur, next, a, rr[a]);
      std::swap(cur, next);
    }
    for (int a = 2; a >= 0; a--) {
      if (rr[a] == 0) continue;
      if (a == 0) {
        ext_adj(R, vol, cur, grad_vol, 0, rr[0]);
      } else {
        cudaMemsetAsync(next, 0, R.N * sizeof(float2), st);
        ext_adj(R, R.pair(a == 1 ? S_MM1 : S_MM2), cur, reinterpret_cast<float *>(next), a, rr[a]);
        std::swap(cur, next);
      }
    }
    if (rr[0] == 0) KLAUNCH("k_soft_add", st, (k_soft_add<<<nb, 256, 0, st>>>(grad_vol, cur, R.N)));
  }
  HDOG_CUDA_TRY(cudaGetLastError());
  return HDOG_OK;
}

}  // namespace hdog
