// norm.cu -- intensity normalization and the regional-erosion operator, sm_103a.
//
// Reference: src/3D/NormalizeFilter.cu (Normalize3DFilter :603-654) and
// src/3D/Erosion3DFilter.cu (Erosion3DFilter :260-268).
//
//   ero  = min over a (2rxy+1)^2 (2rz+1) box, dil = max over it    (nearest border)
//   ero_l = box mean of ero, dil_l = box mean of dil                 (nearest border)
//   norm = I >= min_intensity ? (I - ero_l) / (dil_l - ero_l) : 0
//
// Min and max are exact, so they run in whatever order is cheapest; the box means must
// round exactly like the reference, whose passes go x -> y -> z and each is the
// sequential float sum `val = 0; for j in 0..2r: val += s[j]` times 1.0f/(2r+1).
// Five passes, each one read and one write of the volume:
//
//   mm_z      uint16 -> packed u32     van Herk / Gil-Werman z window in registers
//   mm_y      u32 -> u32               column window from short blocks (window.cuh)
//   mm_x_box  u32 -> float2            row window from short blocks, then the x box
//                                      sum as exact integer sliding sums (2r+1 <= 256:
//                                      every partial sum of the reference's float chain
//                                      is an integer below 2^24, hence exact)
//   box_y     float2 -> float2         the literal y chain, erosion and dilation side by
//                                      side, K outputs per thread from a register window
//   box_z_norm float2 + uint16 -> float the literal z chain fused with the normalization
//
// Erosion and dilation travel as one packed u32 per voxel: low half the running min,
// high half 65535 minus the running max, so one __vminu2 combines both.
#include <algorithm>
#include <climits>

#include "kernels.cuh"
#include "window.cuh"

namespace hdog {

// pack_mm(0, 0): the value a zero-border position contributes
constexpr uint32_t kZeroPacked = 0xFFFF0000u;

// ---------------------------------------------------------------- z pass (min/max)
// VEC consecutive positions of the slice plane per thread (VEC 4: one 8-byte load of
// four uint16 per slice).  Slices at or past depth_valid read as zero (the zero tail
// HDoG3D_main.cpp:166-169 writes for a short last substack).  BORDER: 0 nearest
// (normalization), 1 zero (erosion operator).
template <int BORDER, int VEC>
__global__ void __launch_bounds__(256) k_mm_z(const Sub *subs, int rz, uint32_t *mm) {
  const Sub S = subs[blockIdx.y];
  const int64_t plane = (int64_t)S.W * S.H;
  const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (p >= plane) return;
  const int D = S.D, dv = S.depth_valid;
  const uint16_t *src = S.src + p;
  uint32_t *out = mm + S.vox + p;
  for (int z = 0; z < D; z++) {
    int lo = z - rz, hi = z + rz;
    // nearest border repeats the edge slice (no new value); a zero border, or a slice
    // of the zero tail inside the window, adds a 0
    bool zero = BORDER == 1 && (lo < 0 || hi >= D);
    lo = max(lo, 0);
    hi = min(hi, D - 1);
    if (hi >= dv) zero = true;
    hi = min(hi, dv - 1);
    const uint16_t *q = src + (int64_t)lo * plane;
    if (VEC == 4) {
      uint32_t mn0 = 0xFFFFFFFFu, mn1 = 0xFFFFFFFFu, mx0 = 0u, mx1 = 0u;
      for (int zz = lo; zz <= hi; zz++, q += plane) {
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(q));
        mn0 = __vminu2(mn0, v.x);
        mx0 = __vmaxu2(mx0, v.x);
        mn1 = __vminu2(mn1, v.y);
        mx1 = __vmaxu2(mx1, v.y);
      }
      if (zero) { mn0 = 0u; mn1 = 0u; }
      const uint32_t n0 = ~mx0, n1 = ~mx1;
      uint4 o;
      o.x = __byte_perm(mn0, n0, 0x5410);
      o.y = __byte_perm(mn0, n0, 0x7632);
      o.z = __byte_perm(mn1, n1, 0x5410);
      o.w = __byte_perm(mn1, n1, 0x7632);
      *reinterpret_cast<uint4 *>(out + (int64_t)z * plane) = o;
    } else {
      uint32_t mn = 0xFFFFu, mx = 0u;
      for (int zz = lo; zz <= hi; zz++, q += plane) {
        const uint32_t v = __ldg(q);
        mn = min(mn, v);
        mx = max(mx, v);
      }
      out[(int64_t)z * plane] = pack_mm(zero ? 0u : mn, mx);
    }
  }
}

// The same z pass with a compile-time radius, streaming van Herk / Gil-Werman in registers: a
// thread owns VEC neighbouring columns (two where the slices' 4-byte words hold two columns each)
// and runs down z, every input slice loaded once (the windowed loop above reads each one 2R+1
// times).  A voxel is packed as (v, 65535 - v), so one __vminu2 carries the min and the max.
template <int R, int BORDER, int VEC>
__global__ void __launch_bounds__(128) k_mm_z_stream(const Sub *subs, uint32_t *mm) {
  constexpr int L = 2 * R + 1;
  const Sub S = subs[blockIdx.y];
  const int64_t plane = (int64_t)S.W * S.H;
  const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
  if (p >= plane) return;
  const int D = S.D, dv = S.depth_valid;
  const uint16_t *col = S.src + p;
  uint32_t *oc = mm + S.vox + p;
  struct Cols {
    uint32_t c[VEC];
  };
  auto ld = [&](int z) -> Cols {
    Cols r;
    const bool out = BORDER == 1 && (z < 0 || z >= D);
    z = clampi(z, 0, D - 1);
    if (out || z >= dv) {
#pragma unroll
      for (int k = 0; k < VEC; k++) r.c[k] = kZeroPacked;
    } else if constexpr (VEC == 2) {
      const uint32_t v = __ldg(reinterpret_cast<const uint32_t *>(col + (int64_t)z * plane));
      r.c[0] = __byte_perm(v, ~v, 0x5410);
      r.c[1] = __byte_perm(v, ~v, 0x7632);
    } else {
      const uint32_t v = __ldg(col + (int64_t)z * plane);
      r.c[0] = __byte_perm(v, ~v, 0x5410);
    }
    return r;
  };
  auto vmin = [](Cols a, Cols b) {
    Cols r;
#pragma unroll
    for (int k = 0; k < VEC; k++) r.c[k] = __vminu2(a.c[k], b.c[k]);
    return r;
  };
  Cols suf[L], cur[L];
#pragma unroll
  for (int j = 0; j < L; j++) suf[j] = ld(j - R);
#pragma unroll
  for (int j = L - 2; j >= 0; j--) suf[j] = vmin(suf[j], suf[j + 1]);
  for (int t0 = 0; t0 < D; t0 += L) {
#pragma unroll
    for (int j = 0; j < L; j++) cur[j] = ld(t0 - R + L + j);
    Cols pre;
#pragma unroll
    for (int k = 0; k < VEC; k++) pre.c[k] = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < L; i++) {
      const Cols m = i == 0 ? suf[0] : vmin(suf[i], pre);
      if (t0 + i < D) {
        uint32_t *o = oc + (int64_t)(t0 + i) * plane;
        if constexpr (VEC == 2) *reinterpret_cast<uint2 *>(o) = make_uint2(m.c[0], m.c[1]);
        else *o = m.c[0];
      }
      pre = vmin(pre, cur[i]);
    }
    suf[L - 1] = cur[L - 1];
#pragma unroll
    for (int j = L - 2; j >= 0; j--) suf[j] = vmin(cur[j], suf[j + 1]);
  }
}

// Van Herk / Gil-Werman over blocks of L entries of a smem line: g = running min from
// each block's start (written to G), h = running min to each block's end (written over
// A).  The window [t, t + L - 1] is then min(h[t], g[t + L - 1]).
__device__ __forceinline__ void vhgw_chain(uint32_t *A, uint32_t *G, int i0, int i1, int step) {
  uint32_t run = 0xFFFFFFFFu;
  for (int i = i0; i < i1; i++) {
    run = __vminu2(run, A[i * step]);
    G[i * step] = run;
  }
  run = 0xFFFFFFFFu;
  for (int i = i1 - 1; i >= i0; i--) {
    run = __vminu2(run, A[i * step]);
    A[i * step] = run;
  }
}

// ---------------------------------------------------------------- y pass (min/max)
// A block owns 32 columns x ty output rows of one slice; it stages rows
// [y0 - r, y0 + ty + r) (border rule applied) and runs one chain per (column, block).
template <int BORDER>
__global__ void __launch_bounds__(256) k_mm_y(const Sub *subs, int r, int ty, const uint32_t *in, uint32_t *out) {
  extern __shared__ uint32_t smy[];
  const Sub S = subs[blockIdx.y];
  const int W = S.W, H = S.H;
  const int tx_n = (W + 31) / 32, ty_n = (H + ty - 1) / ty;
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)tx_n * ty_n * S.D) return;
  const int z = (int)(bid / ((int64_t)tx_n * ty_n));
  const int rem = (int)(bid % ((int64_t)tx_n * ty_n));
  const int x0 = (rem % tx_n) * 32, y0 = (rem / tx_n) * ty;
  const int L = 2 * r + 1, n0 = ty + 2 * r;
  uint32_t *A = smy, *G = smy + n0 * 32;
  const int c = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int x = x0 + c;
  const bool xin = x < W;
  const uint32_t *sl = in + S.vox + (int64_t)z * W * H + (xin ? x : 0);
  for (int i = w; i < n0; i += nw) {
    const int y = y0 - r + i;
    uint32_t v;
    if (BORDER == 1 && (y < 0 || y >= H)) v = kZeroPacked;
    else v = sl[(int64_t)clampi(y, 0, H - 1) * W];
    A[i * 32 + c] = v;
  }
  __syncthreads();
  const int nb = (n0 + L - 1) / L;
  for (int b = w; b < nb; b += nw) vhgw_chain(A + c, G + c, b * L, min(b * L + L, n0), 32);
  __syncthreads();
  if (!xin) return;
  uint32_t *o = out + S.vox + (int64_t)z * W * H + x;
  const int tn = min(ty, H - y0);
  for (int t = w; t < tn; t += nw) o[(int64_t)(y0 + t) * W] = __vminu2(A[t * 32 + c], G[(t + 2 * r) * 32 + c]);
}

// ---------------------------------------------------------------- x pass (min/max + box)
// A block owns ry rows x tx outputs.  MODE 0: min/max window, then the exact x box sum
// -> float2 (ero_x, dil_x); MODE 1: min window only -> uint16 (erosion result); MODE 2:
// min/max window only -> packed u32 (followed by the float-chain box for 2r+1 > 256).
constexpr int kBoxC = 16;   // box outputs per thread (sliding integer sums)

template <int BORDER, int MODE>
__global__ void __launch_bounds__(256) k_mm_x(const Sub *subs, int r, int ry, int tx, const uint32_t *in,
                                              void *out) {
  extern __shared__ uint32_t smx[];
  const Sub S = subs[blockIdx.y];
  const int W = S.W;
  const int64_t rows = (int64_t)S.H * S.D;
  const int segs = (W + tx - 1) / tx;
  const int64_t bid = blockIdx.x;
  if (bid >= ((rows + ry - 1) / ry) * segs) return;
  const int64_t row0 = (bid / segs) * ry;
  const int x0 = (int)(bid % segs) * tx;
  const int hm = MODE == 0 ? r : 0;            // halo of the min/max result the box needs
  const int n0 = tx + 2 * hm + 2 * r;          // staged entries per row
  const int stride = n0 | 1;                   // odd: chains of neighbouring rows hit distinct banks
  uint32_t *A = smx, *G = smx + ry * stride;
  const int base = x0 - hm - r;                // x of A[row][0]
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  for (int rl = w; rl < ry; rl += nw) {
    const int64_t row = min(row0 + rl, rows - 1);
    const uint32_t *line = in + S.vox + row * W;
    for (int i = lane; i < n0; i += 32) {
      const int xx = base + i;
      uint32_t v;
      if (BORDER == 1 && (xx < 0 || xx >= W)) v = kZeroPacked;
      else v = line[clampi(xx, 0, W - 1)];
      A[rl * stride + i] = v;
    }
  }
  __syncthreads();
  const int L = 2 * r + 1;
  const int nb = (n0 + L - 1) / L;
  for (int ch = tid; ch < ry * nb; ch += blockDim.x) {
    const int rl = ch % ry, b = ch / ry;
    vhgw_chain(A + rl * stride, G + rl * stride, b * L, min(b * L + L, n0), 1);
  }
  __syncthreads();
  const int tn = min(tx, W - x0);
  if (MODE != 0) {
    for (int rl = w; rl < ry; rl += nw) {
      const int64_t row = row0 + rl;
      if (row >= rows) break;
      for (int k = lane; k < tn; k += 32) {
        const uint32_t m = __vminu2(A[rl * stride + k], G[rl * stride + k + 2 * r]);
        if (MODE == 1) reinterpret_cast<uint16_t *>(out)[S.vox + row * W + x0 + k] = (uint16_t)(m & 0xFFFFu);
        else reinterpret_cast<uint32_t *>(out)[S.vox + row * W + x0 + k] = m;
      }
    }
    return;
  }
  // m at x = x0 - r + k (nearest border: positions outside the row take the edge value)
  const int nm = tx + 2 * r, mstride = nm | 1;
  uint32_t *M = G + ry * stride;
  for (int rl = w; rl < ry; rl += nw)
    for (int k = lane; k < nm; k += 32) {
      const int kc = clampi(x0 - r + k, 0, W - 1) - (x0 - r);
      M[rl * mstride + k] = __vminu2(A[rl * stride + kc], G[rl * stride + kc + 2 * r]);
    }
  __syncthreads();
  // sliding sums, C outputs per thread; results staged (over A and G) for coalesced stores
  float2 *stage = reinterpret_cast<float2 *>(smx);
  const int sstride = tx + 1;
  const float inv = 1.0f / (float)L;
  const uint32_t full = (uint32_t)L * 0xFFFFu;
  const int nchunks = tx / kBoxC;
  for (int ch = tid; ch < ry * nchunks; ch += blockDim.x) {
    const int rl = ch % ry, c0 = (ch / ry) * kBoxC;
    const uint32_t *m = M + rl * mstride + c0;
    uint32_t slo = 0, shi = 0;
    for (int j = 0; j < L; j++) {
      const uint32_t v = m[j];
      slo += v & 0xFFFFu;
      shi += v >> 16;
    }
    float2 res[kBoxC];
#pragma unroll
    for (int t = 0; t < kBoxC; t++) {
      res[t] = make_float2((float)slo * inv, (float)(full - shi) * inv);
      if (t + 1 < kBoxC) {
        const uint32_t vn = m[t + L], vo = m[t];
        slo += (vn & 0xFFFFu) - (vo & 0xFFFFu);
        shi += (vn >> 16) - (vo >> 16);
      }
    }
    // A and G are free once M is built: the stage overwrites them while M is still read
#pragma unroll
    for (int t = 0; t < kBoxC; t++) stage[rl * sstride + c0 + t] = res[t];
  }
  __syncthreads();
  float2 *o = reinterpret_cast<float2 *>(out);
  for (int rl = w; rl < ry; rl += nw) {
    const int64_t row = row0 + rl;
    if (row >= rows) break;
    for (int k = lane; k < tn; k += 32) o[S.vox + row * W + x0 + k] = stage[rl * sstride + k];
  }
}

// ---------------------------------------------------------------- reaches below 4
// Windows of at most seven entries are folded in registers: they are shorter than the blocks of the passes below, and
// chains in shared memory cost more than their few mins.  HBM-bound.  2560x2160x16, reaches 1 to 3: y 215 -> 119 to
// 137 us.  640x720x32 erosion at reach 2: y 54 -> 25 us, x 45 -> 17.  (The x box of these reaches and rows of other
// widths stay with k_mm_x: a load an entry and an output takes 410 to 790 us where it takes 380.)
template <int BORDER>
__device__ __forceinline__ uint32_t mm_at(const uint32_t *line, int i, int n, int64_t step) {
  return BORDER == 1 && (i < 0 || i >= n) ? kZeroPacked : __ldg(line + clampi(i, 0, n - 1) * step);
}

// A warp takes kShortRows rows of 32 columns.
constexpr int kShortRows = 8;
template <int BORDER, int R>
__global__ void __launch_bounds__(256) k_mm_y_short(const Sub *subs, const uint32_t *in, uint32_t *out) {
  const Sub S = subs[blockIdx.y];
  const int W = S.W, H = S.H, tx_n = (W + 31) / 32, ty_n = (H + 8 * kShortRows - 1) / (8 * kShortRows);
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)tx_n * ty_n * S.D) return;
  const int z = (int)(bid / ((int64_t)tx_n * ty_n)), rem = (int)(bid % ((int64_t)tx_n * ty_n));
  const int x = (rem % tx_n) * 32 + (threadIdx.x & 31), y0 = ((rem / tx_n) * 8 + (threadIdx.x >> 5)) * kShortRows;
  if (x >= W || y0 >= H) return;
  const int64_t sl = S.vox + (int64_t)z * W * H + x;
  uint32_t v[kShortRows + 2 * R];
#pragma unroll
  for (int j = 0; j < kShortRows + 2 * R; j++) v[j] = mm_at<BORDER>(in + sl, y0 - R + j, H, W);
#pragma unroll
  for (int k = 0; k < kShortRows; k++) {
    uint32_t m = v[k];
#pragma unroll
    for (int j = 1; j <= 2 * R; j++) m = __vminu2(m, v[k + j]);
    if (y0 + k < H) out[sl + (int64_t)(y0 + k) * W] = m;
  }
}

// The erosion's x pass on rows of whole, aligned quads: a thread reads its quad and the two beside it.
template <int R>
__global__ void __launch_bounds__(256) k_erode_x_quad(const Sub *subs, const uint32_t *in, uint16_t *out) {
  const Sub S = subs[blockIdx.y];
  const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 4;
  if (i >= (int64_t)S.W * S.H * S.D) return;
  const int x = (int)((uint32_t)i % (uint32_t)S.W);
  const uint4 *p = reinterpret_cast<const uint4 *>(in + S.vox + i);
  const uint4 zero = make_uint4(kZeroPacked, kZeroPacked, kZeroPacked, kZeroPacked);
  const uint4 c = __ldg(p), a = x > 0 ? __ldg(p - 1) : zero, b = x + 4 < S.W ? __ldg(p + 1) : zero;
  const uint32_t v[12] = {a.x, a.y, a.z, a.w, c.x, c.y, c.z, c.w, b.x, b.y, b.z, b.w};
  uint32_t m[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    m[k] = v[4 + k - R];
#pragma unroll
    for (int j = 1 - R; j <= R; j++) m[k] = __vminu2(m[k], v[4 + k + j]);
  }
  *reinterpret_cast<uint2 *>(out + S.vox + i) = make_uint2(__byte_perm(m[0], m[1], 0x5410), __byte_perm(m[2], m[3], 0x5410));
}

// ---------------------------------------------------------------- y / x passes for any reach
// Windows from short blocks (window.cuh), for reaches from 4 up.
struct PackedMin {
  typedef uint32_t T;
  __device__ __forceinline__ static T op(T a, T b) { return __vminu2(a, b); }
};

constexpr int kColWarps = 8;

// y pass: a block of 32 columns x kColWarps warps runs down `seg` rows of one slice, B rows per warp
// and step, every input row read once (the 2r halo rows twice per segment).
// HBM and latency: at reach 20 67% of the DRAM cycles at 28 warps per SM.  2560x2160x32 substacks:
// eight with reach 20 2.16 -> 1.89 ms (against columns of 41 entries in registers), four with reach
// 100 9.26 -> 1.33 ms (against chains of 201 in shared memory).
template <int BORDER, int B>
__global__ void __launch_bounds__(32 * kColWarps) k_mm_y_cols(const Sub *subs, int r, int seg, const uint32_t *in,
                                                              uint32_t *out) {
  extern __shared__ uint32_t ring_y[];
  const Sub S = subs[blockIdx.z];
  const int W = S.W, H = S.H;
  const int nseg = (H + seg - 1) / seg;
  const int z = blockIdx.y / nseg, ys = (blockIdx.y % nseg) * seg;
  if (z >= S.D) return;
  const int x = blockIdx.x * 32 + threadIdx.x, n = min(seg, H - ys);
  const bool xin = x < W;
  const int64_t base = S.vox + (int64_t)z * W * H + min(x, W - 1);
  const uint32_t *col = in + base;
  uint32_t *oc = out + base + (int64_t)ys * W;
  ext_cols<PackedMin, B, kColWarps>(
      ring_y, n, r,
      [&](int a, uint32_t (&v)[B]) {
        const int y = ys - r + a;
        if (y >= 0 && y + B <= H) {
          const uint32_t *p = col + (int64_t)y * W;
#pragma unroll
          for (int j = 0; j < B; j++, p += W) v[j] = __ldg(p);
        } else {
#pragma unroll
          for (int j = 0; j < B; j++) {
            const bool zero = BORDER == 1 && (y + j < 0 || y + j >= H);
            v[j] = zero ? kZeroPacked : __ldg(col + (int64_t)clampi(y + j, 0, H - 1) * W);
          }
        }
      },
      [&](int t, uint32_t m) {
        if (xin) oc[(int64_t)t * W] = m;
      });
}

// x pass, G lanes per row, outputs as k_mm_x's MODE: 0 the exact x box sums of the extremes -> float2
// (2r + 1 <= 255), 1 the min -> uint16, 2 the packed extremes.  A lane's 8 neighbours are loaded as
// one 32-byte word and its 8 box means stored as two where the addresses allow it: the row starts `pad`
// entries early, so that for even reaches inputs and outputs both fall on 32 bytes (for odd ones the
// outputs do, and the inputs on 8).  The next chunk's inputs are loaded before this one is worked on.
// MODE 0: a lane's first box sum is the difference of two prefix sums of the extremes (a scan of
// the lanes' totals, and the prefix at the one place of a block where its windows start, from the lane
// that many blocks back); the other seven slide, taking the extremes that leave from a second ring. All in
// wrapping integers; the row's first and last extreme stand for the positions outside it.
// G = 8 (row_of_8): chunks of 64 entries waste less of a short row, and the scan is three steps.
// Bound by instruction issue and the shared-memory pipe.
// 2560x2160x32 substacks: eight with reach 20 3.85 -> 3.41 ms (against rows of 41 entries in
// registers), four with reach 100 9.85 -> 1.62 ms (against chains of 201 in shared memory); 256x256
// and half frames with reach 20 83 -> 59 us a batch.
constexpr int kRowWarps = 4;

// 32-byte global accesses (sm_100 on)
__device__ __forceinline__ void ld8(const uint32_t *p, uint32_t (&v)[8]) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
      : "l"(p));
}
__device__ __forceinline__ void st8(float2 *p, float2 a, float2 b, float2 c, float2 d) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y),
               "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y)
               : "memory");
}
// acc +- one half of a packed pair
template <int HALF, int SIGN>
__device__ __forceinline__ uint32_t add_half(uint32_t pair, uint32_t acc) {
  int r;
  asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(r) : "r"(pair), "r"((SIGN & 0xFF) << (8 * HALF)), "r"((int)acc));
  return (uint32_t)r;
}

template <int BORDER, int MODE, int G, int Q>
__global__ void __launch_bounds__(32 * kRowWarps) k_mm_x_rows(const Sub *subs, int r, const uint32_t *in, void *out) {
  using R = RowRing<G>;
  __shared__ uint32_t smr[kRowWarps][R::WORDS * (MODE == 0 ? 2 : 1)];
  const Sub S = subs[blockIdx.y];
  const int W = S.W, gl = threadIdx.x & (G - 1), w = threadIdx.x >> 5;
  const int64_t rows = (int64_t)S.H * S.D;
  const int64_t row0 = ((int64_t)blockIdx.x * kRowWarps + w) * R::LINES;
  if (row0 >= rows) return;
  const int64_t mine = row0 + (threadIdx.x & 31) / G, row = min(mine, rows - 1);
  const bool live = mine < rows;
  uint32_t *suf = smr[w], *ring = suf + R::WORDS;   // ring: MODE 0, the extremes
  const uint32_t *line = in + S.vox + row * W;
  const int n_in = W + 2 * r, n_e = MODE == 0 ? W + 3 * r : n_in;
  const int L = 2 * r + 1;
  const float inv = 1.0f / (float)L;
  const uint32_t full = (uint32_t)L * 0xFFFFu;
  constexpr int QP = Q == 0 ? 7 : Q - 1;            // 8 ceil(L / 8) - L
  const int backp = (L + 7) / 8;
  // entry e is position e - r; entries -pad .. -1 are there for the alignment only
  const uintptr_t in0 = reinterpret_cast<uintptr_t>(line - r);
  float2 *o2 = reinterpret_cast<float2 *>(out) + S.vox + row * W;
  const uintptr_t out0 = reinterpret_cast<uintptr_t>(o2 - 3 * r);
  const int pad = MODE != 0 ? 0 : Q % 4 == 0 ? (int)((in0 >> 2) & 7) : (int)((out0 >> 3) & 3);
  const int in_al = (int)(((in0 >> 2) - pad) & 7);
  const bool out_al = (((out0 >> 3) - pad) & 3) == 0;
  uint32_t nv[8], hist[6] = {0, 0, 0, 0, 0, 0};
  uint32_t m0 = 0, mlast = 0, clo = 0, chi = 0, plo = 0, phi = 0;
  auto fetch = [&](int c) {
    const int x = c + 8 * gl - r;
    const uint32_t *p = line + x;
    if (x >= 0 && x + 8 <= W && (in_al & 1) == 0) {
      if (in_al == 0) {
        ld8(p, nv);
      } else {
#pragma unroll
        for (int o = 0; o < 8; o += 2) {
          const uint2 a = __ldg(reinterpret_cast<const uint2 *>(p + o));
          nv[o] = a.x;
          nv[o + 1] = a.y;
        }
      }
    } else {
#pragma unroll
      for (int o = 0; o < 8; o++)
        nv[o] = (BORDER == 1 && (x + o < 0 || x + o >= W)) ? kZeroPacked : __ldg(line + clampi(x + o, 0, W - 1));
    }
  };
  int c = -pad;   // the chunk's first entry; the warp's rows may differ by up to 7
  fetch(c);
  int pc = 0;
  for (int i = 0; i < n_e + (MODE == 0 ? 7 : 0); i += R::CHUNK, c += R::CHUNK) {
    uint32_t v[8], m[8];
#pragma unroll
    for (int o = 0; o < 8; o++) v[o] = nv[o];
    if (i < n_in) fetch(c + R::CHUNK);
    ext_row_chunk<PackedMin, G, Q>(suf, pc, r, v, hist, m);
    const int e0 = c + 8 * gl;   // the window that ends with entry e is centred on position e - 2r
    if (MODE == 0) {
      const int ef = 2 * r, el = W - 1 + 2 * r;   // the first and the last position's entries
      const bool inside = __all_sync(0xFFFFFFFFu, c >= ef + L && c + R::CHUNK - 1 < el);
      if (!inside) {
        uint32_t tf = m[0], tl = m[0];
#pragma unroll
        for (int o = 1; o < 8; o++) {
          tf = o == ((ef - c) & 7) ? m[o] : tf;
          tl = o == ((el - c) & 7) ? m[o] : tl;
        }
        tf = __shfl_sync(0xFFFFFFFFu, tf, ((ef - c) >> 3) & (G - 1), G);
        tl = __shfl_sync(0xFFFFFFFFu, tl, ((el - c) >> 3) & (G - 1), G);
        if (ef >= c && ef < c + R::CHUNK) m0 = tf;
        if (el >= c && el < c + R::CHUNK) mlast = tl;
        // left of the row: nothing here, the first extreme's share comes with the box; right of it: the last extreme
#pragma unroll
        for (int o = 0; o < 8; o++) m[o] = e0 + o < ef ? 0u : e0 + o > el ? mlast : m[o];
      }
      const RowAt<G> at(pc);
      const int own = at(0);
      uint32_t tlo = 0, thi = 0, qlo = 0, qhi = 0;
#pragma unroll
      for (int o = 0; o < 8; o++) {
        ring[o * R::PITCH + own] = m[o];
        tlo = add_half<0, 1>(m[o], tlo);
        thi = add_half<1, 1>(m[o], thi);
        if (o == QP) {
          qlo = tlo;
          qhi = thi;
        }
      }
      uint32_t blo = tlo, bhi = thi;   // inclusive scan of the lanes' totals
#pragma unroll
      for (int d = 1; d < G; d <<= 1) {
        const uint32_t a = __shfl_up_sync(0xFFFFFFFFu, blo, d, G), b = __shfl_up_sync(0xFFFFFFFFu, bhi, d, G);
        if (gl >= d) {
          blo += a;
          bhi += b;
        }
      }
      const uint32_t slo = __shfl_sync(0xFFFFFFFFu, blo, G - 1, G), shi = __shfl_sync(0xFFFFFFFFu, bhi, G - 1, G);
      blo += clo - tlo;   // the sum before the lane
      bhi += chi - thi;
      clo += slo;
      chi += shi;
      qlo += blo;         // the prefix at the place where windows start
      qhi += bhi;
      uint32_t a = blo - row_lag<G>(qlo, plo, backp), d = bhi - row_lag<G>(qhi, phi, backp);
      plo = qlo;
      phi = qhi;
      __syncwarp();
      const uint32_t *p0 = ring + at(backp), *p1 = ring + at(backp - 1);
      if (!inside) {
        const uint32_t left = (uint32_t)max(0, 4 * r - e0);   // positions of the box left of the row
        a += left * (m0 & 0xFFFFu);
        d += left * (m0 >> 16);
      }
      a = add_half<0, 1>(m[0], a);
      d = add_half<1, 1>(m[0], d);
      float2 res[8];
#pragma unroll
      for (int o = 0; o < 8; o++) {
        if (o) {
          uint32_t x = QP + o < 8 ? p0[(QP + o) * R::PITCH] : p1[(QP + o - 8) * R::PITCH];
          if (!inside) x = e0 + o - L < ef ? m0 : x;
          a = add_half<0, -1>(x, add_half<0, 1>(m[o], a));
          d = add_half<1, -1>(x, add_half<1, 1>(m[o], d));
        }
        res[o] = make_float2((float)a * inv, (float)(full - d) * inv);
      }
      const int u = e0 - 3 * r;
      if (live) {
        if (out_al && u >= 0 && u + 8 <= W) {
          st8(o2 + u, res[0], res[1], res[2], res[3]);
          st8(o2 + u + 4, res[4], res[5], res[6], res[7]);
        } else {
#pragma unroll
          for (int o = 0; o < 8; o++)
            if (u + o >= 0 && u + o < W) o2[u + o] = res[o];
        }
      }
    } else if (live) {
      const int u = e0 - 2 * r;
#pragma unroll
      for (int o = 0; o < 8; o++) {
        if (u + o < 0 || u + o >= W) continue;
        if (MODE == 1) reinterpret_cast<uint16_t *>(out)[S.vox + row * W + u + o] = (uint16_t)(m[o] & 0xFFFFu);
        else reinterpret_cast<uint32_t *>(out)[S.vox + row * W + u + o] = m[o];
      }
    }
    __syncwarp();   // the rings' oldest blocks are rewritten next chunk
    pc += G;
    if (pc >= R::NB) pc = 0;
  }
}

// ---------------------------------------------------------------- x pass (box, float chain)
// The literal float chain of the x box for windows wider than 256 (where the partial
// sums stop being exact integers), over a packed min/max volume.
__global__ void k_box_x_chain(const Sub *subs, int r, const uint32_t *in, float2 *out) {
  extern __shared__ float2 sfx[];
  constexpr int kSeg = 256;
  const Sub S = subs[blockIdx.y];
  const int segs = (S.W + kSeg - 1) / kSeg;
  const int64_t rows = (int64_t)S.H * S.D;
  const int64_t bid = blockIdx.x;
  if (bid >= rows * segs) return;
  const int64_t row = bid / segs;
  const int x0 = (int)(bid % segs) * kSeg;
  const int L = 2 * r + 1, n0 = kSeg + 2 * r;
  const float inv = 1.0f / (float)L;
  const uint32_t *line = in + S.vox + row * S.W;
  for (int i = threadIdx.x; i < n0; i += blockDim.x) {
    const uint32_t v = line[clampi(x0 - r + i, 0, S.W - 1)];
    sfx[i] = make_float2((float)mm_lo(v), (float)mm_hi(v));
  }
  __syncthreads();
  const int x = x0 + threadIdx.x;
  if (x >= S.W) return;
  float2 acc = make_float2(0.f, 0.f);
  for (int j = 0; j < L; j++) acc = add2(acc, sfx[threadIdx.x + j]);
  out[S.vox + row * S.W + x] = mul2(acc, make_float2(inv, inv));
}

// ---------------------------------------------------------------- y / z passes (box mean)
// The y box chain with a compile-time window: K outputs from a window of K registers
// (input j + k feeds output k at step j, in the reference's order: 0 + s0 + s1 + ...).
template <int K, int L, class LoadF>
__device__ __forceinline__ void box_chain_t(LoadF load, float2 (&acc)[K]) {
  float2 win[K];
#pragma unroll
  for (int k = 0; k < K; k++) {
    win[k] = load(k);
    acc[k] = make_float2(0.f, 0.f);
  }
#pragma unroll
  for (int j = 0; j < L; j++) {
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] = add2(acc[k], win[(j + k) % K]);
    if (j + K < L + K - 1) win[j % K] = load(j + K);
  }
}

// K outputs of a column per thread: a window of K inputs moves through registers, (K + 2r) loads for K (2r + 1) f32x2
// adds.  The adds are the reference's chains and cannot be shared, so at long reaches the FMA pipe is the bound (reach
// 100: 7.6 ms of adds in 8.4) and at short ones HBM; running pointers keep the address arithmetic out of it.  2560 x 2160
// x 16 at reach 16: K = 12 305 us, 16 273, 20 304; reach 64: 760, 720, 718; reach 127: 1421, 1372, 1337.

template <int K>
__global__ void __launch_bounds__(128) k_box_y(const Sub *subs, int r, const float2 *in, float2 *out) {
  const Sub S = subs[blockIdx.y];
  const int rows_per_blk = blockDim.y * K;
  const int tx_n = (S.W + 31) / 32, ty_n = (S.H + rows_per_blk - 1) / rows_per_blk;
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)tx_n * ty_n * S.D) return;
  const int z = (int)(bid / ((int64_t)tx_n * ty_n));
  const int rem = (int)(bid % ((int64_t)tx_n * ty_n));
  const int x = (rem % tx_n) * 32 + threadIdx.x;
  const int y0 = (rem / tx_n) * rows_per_blk + threadIdx.y * K;
  if (x >= S.W || y0 >= S.H) return;
  const int H = S.H, W = S.W, L = 2 * r + 1;
  const float2 *col = in + S.vox + (int64_t)z * W * H + x;
  float2 acc[K];
  if (y0 - r >= 0 && y0 + K + r <= H) {
    const float2 *p = col + (int64_t)(y0 - r) * W;
    box_chain<K>(L, [&](int) {   // loads its inputs in order
      const float2 v = __ldg(p);
      p += W;
      return v;
    }, acc);
  } else {
    box_chain<K>(L, [&](int i) { return __ldg(col + (int64_t)clampi(y0 - r + i, 0, H - 1) * W); }, acc);
  }
  const float inv = 1.0f / (float)L;
  float2 *o = out + S.vox + (int64_t)z * W * H + x;
#pragma unroll
  for (int k = 0; k < K; k++)
    if (y0 + k < H) o[(int64_t)(y0 + k) * W] = mul2(acc[k], make_float2(inv, inv));
}

// The y box with a compile-time radius: K outputs of one column per thread from a register
// window (box_chain_t), loads and stores walking running pointers, so that no address
// arithmetic joins the f32x2 adds in the FMA pipe.
template <int R, int K>
__global__ void __launch_bounds__(128, 6) k_box_y_t(const Sub *subs, const float2 *in, float2 *out) {
  constexpr int L = 2 * R + 1;
  const Sub S = subs[blockIdx.y];
  const int rows_per_blk = blockDim.y * K;
  const int tx_n = (S.W + 31) / 32, ty_n = (S.H + rows_per_blk - 1) / rows_per_blk;
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)tx_n * ty_n * S.D) return;
  const int z = (int)(bid / ((int64_t)tx_n * ty_n));
  const int rem = (int)(bid % ((int64_t)tx_n * ty_n));
  const int x = (rem % tx_n) * 32 + threadIdx.x;
  const int y0 = (rem / tx_n) * rows_per_blk + threadIdx.y * K;
  if (x >= S.W || y0 >= S.H) return;
  const int H = S.H, W = S.W;
  const float2 *col = in + S.vox + (int64_t)z * W * H + x;
  float2 acc[K];
  if (y0 - R >= 0 && y0 + K + R <= H) {
    const float2 *q = col + (int64_t)(y0 - R) * W;   // box_chain_t loads its inputs in order
    box_chain_t<K, L>([&](int) {
      const float2 v = __ldg(q);
      q += W;
      return v;
    }, acc);
  } else {
    box_chain_t<K, L>([&](int i) { return __ldg(col + (int64_t)clampi(y0 - R + i, 0, H - 1) * W); }, acc);
  }
  const float inv = 1.0f / (float)L;
  float2 *o = out + S.vox + (int64_t)z * W * H + (int64_t)y0 * W + x;
#pragma unroll
  for (int k = 0; k < K; k++, o += W)
    if (y0 + k < H) *o = mul2(acc[k], make_float2(inv, inv));
}

// Where plane position p of slice 0 lies in the normalized volume, whose rows may be padded (PAD).
template <bool PAD>
__device__ __forceinline__ int64_t norm_at(const Sub &S, int64_t p) {
  return PAD ? S.pvox + p + (int64_t)((uint32_t)p / (uint32_t)S.W) * (S.P - S.W) : S.vox + p;
}

// z pass of the box mean fused with Normalize3DKernel (NormalizeFilter.cu:571-586).
constexpr int kBoxZK = 8;

__global__ void __launch_bounds__(128) k_box_z_norm(const Sub *subs, int rz, float min_intensity, const float2 *in,
                                                    float *norm, float *ero_l, float *dil_l) {
  const Sub S = subs[blockIdx.y];
  const int64_t plane = (int64_t)S.W * S.H;
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= plane) return;
  const float2 *col = in + S.vox + p;
  const int D = S.D, L = 2 * rz + 1;
  float *nout = norm + norm_at<true>(S, p);
  const int64_t pplane = (int64_t)S.P * S.H;
  const float inv = 1.0f / (float)L;
  for (int z0 = 0; z0 < D; z0 += kBoxZK) {
    float2 acc[kBoxZK];
    box_chain<kBoxZK>(L, [&](int i) { return __ldg(col + clampi(z0 - rz + i, 0, D - 1) * plane); }, acc);
#pragma unroll
    for (int k = 0; k < kBoxZK; k++) {
      const int z = z0 + k;
      if (z < D) {
        const float2 el = mul2(acc[k], make_float2(inv, inv));
        const float v = z < S.depth_valid ? (float)__ldg(S.src + z * plane + p) : 0.0f;
        nout[z * pplane] = (v >= min_intensity) ? (v - el.x) / (el.y - el.x) : 0.0f;
        if (ero_l) {
          ero_l[S.vox + z * plane + p] = el.x;
          dil_l[S.vox + z * plane + p] = el.y;
        }
      }
    }
  }
}

// The same pass specialised on the z radius: one thread per (column, chunk of kBoxZK slices), every window input loaded
// before the first add so that all loads of a thread are in flight together; neighbouring blocks take the chunks of the
// same columns, which share their overlapping inputs through the caches.  Bound by HBM (14 bytes a voxel) once the
// instructions around the loads are few: chunks whose window lies inside the volume walk two pointers instead of clamping
// and multiplying every index, and ten blocks fit an SM (for which a thread spills 52 bytes at reach 5, 16 at 4).  1.42 G
// voxels at reach 5: 4.23 -> 3.60 ms (5.5 TB/s); chunks of 6 (3.88 ms), 10 (4.48) and 12 (4.42), and a register ring down
// the column (5.9) are slower.  PARTS also stores the box means (stage dumps).
template <int RZ, bool PARTS, bool PAD>
__global__ void __launch_bounds__(128, RZ <= 5 ? 10 : 6) k_box_z_norm_t(const Sub *subs, float min_intensity, const float2 *in,
                                                      float *norm, float *ero_l, float *dil_l) {
  constexpr int L = 2 * RZ + 1, NW = kBoxZK + 2 * RZ;
  const Sub S = subs[blockIdx.y];
  const int plane = S.W * S.H, D = S.D;
  const int nch = (D + kBoxZK - 1) / kBoxZK;
  const int p = (int)(blockIdx.x / nch) * 128 + threadIdx.x;
  const int z0 = (int)(blockIdx.x % nch) * kBoxZK;
  if (p >= plane) return;
  const float2 *col = in + S.vox + p;
  const uint16_t *src = S.src + p;
  float2 win[NW];
  float v[kBoxZK];
  if (z0 >= RZ && z0 + kBoxZK + RZ <= D && z0 + kBoxZK <= S.depth_valid) {
    const float2 *c = col + (int64_t)(z0 - RZ) * plane;
    const uint16_t *s = src + (int64_t)z0 * plane;
#pragma unroll
    for (int i = 0; i < NW; i++) { win[i] = __ldg(c); c += plane; }
#pragma unroll
    for (int k = 0; k < kBoxZK; k++) { v[k] = (float)__ldg(s); s += plane; }
  } else {
#pragma unroll
    for (int i = 0; i < NW; i++) win[i] = __ldg(col + (int64_t)clampi(z0 - RZ + i, 0, D - 1) * plane);
#pragma unroll
    for (int k = 0; k < kBoxZK; k++) {
      const int z = min(z0 + k, D - 1);
      v[k] = z < S.depth_valid ? (float)__ldg(src + (int64_t)z * plane) : 0.0f;
    }
  }
  const float inv = 1.0f / (float)L;
  const int pplane = PAD ? S.P * S.H : plane;
  float *nout = norm + norm_at<PAD>(S, p) + (int64_t)z0 * pplane;
#pragma unroll
  for (int k = 0; k < kBoxZK; k++) {
    float2 acc = make_float2(0.f, 0.f);
#pragma unroll
    for (int j = 0; j < L; j++) acc = add2(acc, win[k + j]);
    const int z = z0 + k;
    if (z < D) {
      const float2 el = mul2(acc, make_float2(inv, inv));
      *nout = (v[k] >= min_intensity) ? (v[k] - el.x) / (el.y - el.x) : 0.0f;
      nout += pplane;
      if (PARTS) {
        ero_l[S.vox + (int64_t)z * plane + p] = el.x;
        dil_l[S.vox + (int64_t)z * plane + p] = el.y;
      }
    }
  }
}

// Copy3DKernel (NormalizeFilter.cu:588-601), used when a normalization radius is 0.
__global__ void k_copy_norm(const Sub *subs, float min_intensity, float *norm) {
  const Sub S = subs[blockIdx.y];
  const int64_t n = (int64_t)S.W * S.H * S.D, plane = (int64_t)S.W * S.H;
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int z = (int)(i / plane);
  const float v = z < S.depth_valid ? (float)S.src[i] : 0.0f;
  norm[norm_at<true>(S, i - z * plane) + (int64_t)z * S.P * S.H] = (v >= min_intensity) ? v : 0.0f;
}

// ---------------------------------------------------------------- launchers
static int max_optin_smem() {
  static const int v = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return n > 0 ? n : 48 * 1024;
  }();
  return v;
}

// The allowance belongs to the kernel, not to the launch, so it is the largest of any call: a smaller one could take
// away what another host thread has just asked for.
template <class F>
static void allow_smem(F *fn, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, max_optin_smem());
}

// vec: the widest of 4, 2, 1 neighbouring columns that the inputs' alignment allows.  The streaming form loads and
// combines whole blocks of 2 rz + 1 slices, two of them at least, so volumes of few slices take the windows' own loads
// (one slice of 2560x2160 at reach 5: 31 against 10 us).
template <int BORDER>
static void mm_z(const Sub *d_subs, int nsub, int plane, int D, int rz, int vec, uint32_t *mm, cudaStream_t s) {
  const dim3 g2(ceil_div(plane / 2, 128), nsub), g1(ceil_div(plane, 128), nsub);
  const int L = 2 * rz + 1;
  switch ((int64_t)D * std::min(D, L) <= 2 * L ? 0 : rz) {
#define HDOG_MMZ_CASE(R)                                                                      \
  case R:                                                                                     \
    if (vec >= 2)                                                                             \
      KLAUNCH("k_mm_z", s, (k_mm_z_stream<R, BORDER, 2><<<g2, 128, 0, s>>>(d_subs, mm)));     \
    else                                                                                      \
      KLAUNCH("k_mm_z", s, (k_mm_z_stream<R, BORDER, 1><<<g1, 128, 0, s>>>(d_subs, mm)));     \
    return;
    HDOG_MMZ_CASE(1) HDOG_MMZ_CASE(2) HDOG_MMZ_CASE(3) HDOG_MMZ_CASE(4)
    HDOG_MMZ_CASE(5) HDOG_MMZ_CASE(6) HDOG_MMZ_CASE(7) HDOG_MMZ_CASE(8)
#undef HDOG_MMZ_CASE
    default:
      break;
  }
  if (vec == 4) {
    dim3 grid(ceil_div(plane / 4, 256), nsub);
    KLAUNCH("k_mm_z", s, (k_mm_z<BORDER, 4><<<grid, 256, 0, s>>>(d_subs, rz, mm)));
  } else {
    dim3 grid(ceil_div(plane, 256), nsub);
    KLAUNCH("k_mm_z", s, (k_mm_z<BORDER, 1><<<grid, 256, 0, s>>>(d_subs, rz, mm)));
  }
}

// Rows per block of the y pass: whole columns when the columns fill the chip, else segments of at
// least one step of the block and one window.
static int mm_y_seg(int64_t cols, int H, int r) {
  const int64_t want = 2048;
  const int64_t nseg = std::max<int64_t>(1, (want + cols - 1) / cols);
  const int seg = (int)std::max<int64_t>(ceil_div(H, nseg), std::max(2 * r, 128));
  return std::min(seg, H);
}

template <int BORDER, int B>
static bool mm_y_cols(const Sub *d_subs, int nsub, int W, int H, int D, int r, const uint32_t *in, uint32_t *out,
                      cudaStream_t s) {
  const int seg = mm_y_seg((int64_t)ceil_div(W, 32) * D * nsub, H, r);
  if ((int64_t)ceil_div(H, seg) * D > 65535) return false;   // the grid's second extent
  const size_t smem = (size_t)ext_cols_rows(r, B, kColWarps) * 32 * sizeof(uint32_t);
  allow_smem(k_mm_y_cols<BORDER, B>, smem);
  const dim3 grid(ceil_div(W, 32), ceil_div(H, seg) * D, nsub);
  KLAUNCH("k_mm_y", s, (k_mm_y_cols<BORDER, B><<<grid, dim3(32, kColWarps), smem, s>>>(d_subs, r, seg, in, out)));
  return true;
}

template <int BORDER>
static void mm_y(const Sub *d_subs, int nsub, int W, int H, int D, int r, const uint32_t *in, uint32_t *out,
                 cudaStream_t s) {
  if (r < 4) {
    const dim3 grid((unsigned)((int64_t)ceil_div(W, 32) * ceil_div(H, 8 * kShortRows) * D), nsub);
    const auto fn = r == 0 ? k_mm_y_short<BORDER, 0> : r == 1 ? k_mm_y_short<BORDER, 1>
                  : r == 2 ? k_mm_y_short<BORDER, 2> : k_mm_y_short<BORDER, 3>;
    KLAUNCH("k_mm_y", s, (fn<<<grid, 256, 0, s>>>(d_subs, in, out)));
    return;
  }
  if (r >= 8 && mm_y_cols<BORDER, 16>(d_subs, nsub, W, H, D, r, in, out, s)) return;
  if (r < 8 && mm_y_cols<BORDER, 8>(d_subs, nsub, W, H, D, r, in, out, s)) return;
  // rows per block: 128, fewer when the staged window would not fit in shared memory
  const int cap_rows = max_optin_smem() / (2 * 32 * 4);
  int ty = 128;
  while (ty > 16 && ty + 2 * r > cap_rows) ty /= 2;
  const size_t smem = (size_t)2 * (ty + 2 * r) * 32 * 4;
  allow_smem(k_mm_y<BORDER>, smem);
  dim3 grid((unsigned)((int64_t)ceil_div(W, 32) * ceil_div(H, ty) * D), nsub);
  KLAUNCH("k_mm_y", s, (k_mm_y<BORDER><<<grid, 256, smem, s>>>(d_subs, r, ty, in, out)));
}

static size_t mm_x_smem(int mode, int r, int ry, int tx) {
  const int hm = mode == 0 ? r : 0;
  const int stride = (tx + 2 * hm + 2 * r) | 1;
  size_t words = (size_t)2 * ry * stride;
  if (mode == 0) {
    words += (size_t)ry * ((tx + 2 * r) | 1);
    words = words > (size_t)ry * (tx + 1) * 2 ? words : (size_t)ry * (tx + 1) * 2;   // staging fits over A + G
  }
  return words * 4;
}

// Whether the tiles of k_mm_x beat a warp a row: a row takes about 0.6 us (erosion 0.5) for each 256 columns, one after
// the other, however few rows there are, and tiles share a long row among many blocks, at a cost per voxel that grows
// with the reach.  us, rows / tiles, at reach 20: 64 rows of 2560 columns 14/12, of 20000 54/15, 608 of 5000 19/25, of
// 20000 62/78; erosion, 256 rows of 20000 51/21, 2160 95/142.
template <int MODE>
static bool mm_x_tiles(int W, int64_t rows, int r) {
  const double by_row = MODE == 0 ? 2.4e-3 : 2.0e-3;                          // us a column
  const double by_voxel = MODE == 0 ? 3.5e-6 + 1e-7 * r : 1.6e-6 + 5e-8 * r;   // us
  return W * (by_row - by_voxel * (double)rows) > 5.0;
}

template <int BORDER, int MODE>
static void mm_x(const Sub *d_subs, int nsub, int W, int64_t rows, int r, const uint32_t *in, void *out,
                 cudaStream_t s) {
  if (MODE == 1 && r < 4 && W % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 7) == 0) {
    const auto fn = r == 0 ? k_erode_x_quad<0> : r == 1 ? k_erode_x_quad<1> : r == 2 ? k_erode_x_quad<2> : k_erode_x_quad<3>;
    KLAUNCH("k_mm_x", s, (fn<<<dim3((unsigned)ceil_div(rows * W / 4, 256), nsub), 256, 0, s>>>(d_subs, in, static_cast<uint16_t *>(out))));
    return;
  }
  if (r >= 4 && r <= (MODE == 0 ? 127 : 255) && !mm_x_tiles<MODE>(W, rows * nsub, r)) {
    switch ((8 - 2 * r % 8) % 8 + (row_of_8(r, W, rows * nsub, MODE == 0 ? INT_MAX : 128) ? 1 : 0)) {
#define HDOG_MMX_CASE(Q)                                                                                     \
  case Q:                                                                                                    \
    KLAUNCH("k_mm_x", s, (k_mm_x_rows<BORDER, MODE, 32, Q><<<dim3(ceil_div(rows, kRowWarps), nsub), 32 * kRowWarps, 0, s>>>( \
                             d_subs, r, in, out)));                                                          \
    return;                                                                                                  \
  case Q + 1:                                                                                                \
    KLAUNCH("k_mm_x", s, (k_mm_x_rows<BORDER, MODE, 8, Q><<<dim3(ceil_div(rows, 4 * kRowWarps), nsub), 32 * kRowWarps, 0, s>>>( \
                             d_subs, r, in, out)));                                                          \
    return;
      HDOG_MMX_CASE(0) HDOG_MMX_CASE(2) HDOG_MMX_CASE(4) HDOG_MMX_CASE(6)
#undef HDOG_MMX_CASE
    }
  }
  // 16 rows x 256 outputs per block, narrower until the staged rows fit in shared
  // memory; MODE 0 runs one thread per (row, chunk of kBoxC outputs).
  int ry = 16, tx = 256;
  while (mm_x_smem(MODE, r, ry, tx) > (size_t)max_optin_smem() && tx > 64) tx /= 2;
  const size_t smem = mm_x_smem(MODE, r, ry, tx);
  const int threads = MODE == 0 ? ry * (tx / kBoxC) : 256;
  allow_smem(k_mm_x<BORDER, MODE>, smem);
  dim3 grid((unsigned)(((rows + ry - 1) / ry) * ceil_div(W, tx)), nsub);
  KLAUNCH("k_mm_x", s, (k_mm_x<BORDER, MODE><<<grid, threads, smem, s>>>(d_subs, r, ry, tx, in, out)));
}

static int mm_z_vec(bool src_aligned8, int plane) { return !src_aligned8 ? 1 : plane % 4 == 0 ? 4 : plane % 2 == 0 ? 2 : 1; }

void launch_normalize(const Sub *d_subs, int nsub, int W, int P, int H, int D, int rxy, int rz, float min_intensity,
                      bool src_aligned8, uint32_t *ma, uint32_t *mb, float2 *fa, float2 *fb, float *norm,
                      cudaStream_t s, float *ero_l, float *dil_l) {
  const int plane = W * H;
  const int64_t rows = (int64_t)H * D;
  mm_z<0>(d_subs, nsub, plane, D, rz, mm_z_vec(src_aligned8, plane), ma, s);
  mm_y<0>(d_subs, nsub, W, H, D, rxy, ma, mb, s);
  if (2 * rxy + 1 <= 256) {
    mm_x<0, 0>(d_subs, nsub, W, rows, rxy, mb, fa, s);
  } else {
    mm_x<0, 2>(d_subs, nsub, W, rows, rxy, mb, ma, s);
    const size_t smem = (size_t)(256 + 2 * rxy) * sizeof(float2);
    allow_smem(k_box_x_chain, smem);
    KLAUNCH("k_box_x_chain", s, (k_box_x_chain<<<dim3((unsigned)(rows * ceil_div(W, 256)), nsub), 256, smem, s>>>(
                                    d_subs, rxy, ma, fa)));
  }
  const int by = 4;
  if (rxy == 20) {   // the workload's radius: compile-time window, 16 outputs a thread
    constexpr int K = 16;
    dim3 gy((unsigned)((int64_t)ceil_div(W, 32) * ceil_div(H, by * K) * D), nsub);
    KLAUNCH("k_box_y", s, (k_box_y_t<20, K><<<gy, dim3(32, by), 0, s>>>(d_subs, fa, fb)));
  } else {
    // fewer outputs a thread, and so more threads, where there are too few to fill the chip
    const int K = (int64_t)W * H * D * nsub < ((int64_t)8 << 20) ? 12 : rxy < 64 ? 16 : 20;
    const auto fn = K == 12 ? k_box_y<12> : K == 16 ? k_box_y<16> : k_box_y<20>;
    dim3 gy((unsigned)((int64_t)ceil_div(W, 32) * ceil_div(H, by * K) * D), nsub);
    KLAUNCH("k_box_y", s, (fn<<<gy, dim3(32, by), 0, s>>>(d_subs, rxy, fa, fb)));
  }
  const dim3 gz(ceil_div(plane, 128) * ceil_div(D, kBoxZK), nsub), bz(128);
  switch (rz) {
#define HDOG_BOXZ_CASE(R)                                                                                   \
  case R:                                                                                                   \
    if (ero_l)                                                                                              \
      KLAUNCH("k_box_z_norm", s, (k_box_z_norm_t<R, true, false><<<gz, bz, 0, s>>>(d_subs, min_intensity, fb, norm, ero_l, dil_l))); \
    else if (P != W)                                                                                        \
      KLAUNCH("k_box_z_norm", s, (k_box_z_norm_t<R, false, true><<<gz, bz, 0, s>>>(d_subs, min_intensity, fb, norm, ero_l, dil_l))); \
    else                                                                                                    \
      KLAUNCH("k_box_z_norm", s, (k_box_z_norm_t<R, false, false><<<gz, bz, 0, s>>>(d_subs, min_intensity, fb, norm, ero_l, dil_l))); \
    break;
    HDOG_BOXZ_CASE(1) HDOG_BOXZ_CASE(2) HDOG_BOXZ_CASE(3) HDOG_BOXZ_CASE(4)
    HDOG_BOXZ_CASE(5) HDOG_BOXZ_CASE(6) HDOG_BOXZ_CASE(7) HDOG_BOXZ_CASE(8)
#undef HDOG_BOXZ_CASE
    default:
      KLAUNCH("k_box_z_norm", s, (k_box_z_norm<<<dim3(ceil_div(plane, 128), nsub), 128, 0, s>>>(
                                     d_subs, rz, min_intensity, fb, norm, ero_l, dil_l)));
  }
}

void launch_copy_norm(const Sub *d_subs, int nsub, int64_t max_n, float min_intensity, float *norm,
                      cudaStream_t s) {
  dim3 grid(ceil_div(max_n, 256), nsub);
  KLAUNCH("k_copy_norm", s, (k_copy_norm<<<grid, 256, 0, s>>>(d_subs, min_intensity, norm)));
}

// Erosion3DFilter: min with a zero border.  Min is separable and exact, so z -> y -> x
// gives the reference's x -> y -> z result.  `tmp` holds two packed u32 volumes.
void launch_erosion(const Sub *d_subs, int nsub, int W, int H, int D, int rxy, int rz, bool src_aligned8,
                    uint32_t *tmp, uint16_t *dst, cudaStream_t s) {
  const int plane = W * H;
  const int64_t n = (int64_t)plane * D;
  uint32_t *a = tmp, *b = tmp + n * nsub;
  mm_z<1>(d_subs, nsub, plane, D, rz, mm_z_vec(src_aligned8, plane), a, s);
  mm_y<1>(d_subs, nsub, W, H, D, rxy, a, b, s);
  mm_x<1, 1>(d_subs, nsub, W, (int64_t)H * D, rxy, b, dst, s);
}

}  // namespace hdog
