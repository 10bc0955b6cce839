// dog.cu -- difference of Gaussians and the Hessian negative-definite mask, sm_103a.
//
// Reference: src/3D/DoG3DFilter.cu (DoG3DFilter :431-437) and
// src/3D/Hessian3DFilter_element.cu (HessianPositiveDefiniteWithElement :355-388).
//
// DoG: both Gaussian scales run together, the small one in the .x lane and the large one
// in the .y lane of an f32x2, so one packed FMA advances both chains.  Each output is the
// reference's chain `sum = 0; for j = -r..r: sum = fma(k[r-j], s[x+j], sum)` with a zero
// border, x then y then z; taps that exist for one scale only run as scalar FMAs on its
// lane, so neither chain sees an extra term.
//
// Hessian: gradients of gradients with a zero halo at every step, computed from a dog
// tile staged in shared memory; only the uint8 mask is written (the six elements are
// written only on request, for stage-wise checks).
#include "kernels.cuh"

namespace hdog {

constexpr int kConvK = 8;       // outputs per thread along y / z

// The passes' intermediate volumes have the rows of the normalized and the DoG volume (pitch P).

// ---------------------------------------------------------------- x pass
// One warp per 128 outputs of a row, staged with the reach on both sides; a lane forms four neighbouring outputs, so
// that a 16-byte shared-memory load brings the inputs of four taps and each tap's coefficient pair
// and duplicated input serve four f32x2 FMAs.
// Instruction-bound (reaches without an unrolled pass, below).  Four 683x517x32 substacks, radii 3 / 5: 460 -> 191 us
// against one output per thread with a shared-memory load per tap.
constexpr int kConvXWarps = 8, kConvXOut = 128;
constexpr int kConvXHalo = 40;   // the widest reach (39), in whole float4

__global__ void __launch_bounds__(32 * kConvXWarps) k_conv_x(const Sub *subs, const __grid_constant__ DogTaps T,
                                                             const float *in, float2 *out) {
  __shared__ __align__(16) float rows_sh[kConvXWarps][kConvXOut + 2 * kConvXHalo + 4];
  const Sub S = subs[blockIdx.y];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = S.W, P = S.P;
  const int segs = (W + kConvXOut - 1) / kConvXOut;
  const int64_t id = (int64_t)blockIdx.x * kConvXWarps + w;
  if (id >= (int64_t)S.H * S.D * segs) return;
  const int64_t row = id / segs;
  const int x0 = (int)(id % segs) * kConvXOut;
  const int ra = T.r[0], rb = T.r[2], rm = max(ra, rb), hx = (rm + 3) & ~3;
  float *sh = rows_sh[w];
  const float *line = in + S.pvox + row * P;
  for (int i = lane; i < kConvXOut + 2 * hx + 4; i += 32) {
    const int x = x0 - hx + i;
    sh[i] = (x >= 0 && x < W) ? line[x] : 0.0f;
  }
  __syncwarp();
  float2 acc[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  const float4 *s4 = reinterpret_cast<const float4 *>(sh) + lane;
  float4 lo = s4[0];
  for (int jb = -hx; jb <= rm; jb += 4) {
    const float4 hi = s4[(jb + hx) / 4 + 1];
    const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    lo = hi;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = jb + u;
      const bool aa = j >= -ra && j <= ra, ab = j >= -rb && j <= rb;
      if (aa && ab) {
        const float2 kk = make_float2(T.k[0][ra - j], T.k[2][rb - j]);
#pragma unroll
        for (int o = 0; o < 4; o++) acc[o] = fma2(kk, make_float2(v[u + o], v[u + o]), acc[o]);
      } else if (ab) {
        const float kk = T.k[2][rb - j];
#pragma unroll
        for (int o = 0; o < 4; o++) acc[o].y = __fmaf_rn(kk, v[u + o], acc[o].y);
      } else if (aa) {
        const float kk = T.k[0][ra - j];
#pragma unroll
        for (int o = 0; o < 4; o++) acc[o].x = __fmaf_rn(kk, v[u + o], acc[o].x);
      }
    }
  }
  const int x = x0 + 4 * lane;
  if (x >= W) return;
  float2 *o = out + S.pvox + row * P + x;
  if ((P & 3) == 0) {   // whole 32-byte sectors; columns past the width are padding
    float4 *o4 = reinterpret_cast<float4 *>(o);
    o4[0] = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
    o4[1] = make_float4(acc[2].x, acc[2].y, acc[3].x, acc[3].y);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (x + k < W) o[k] = acc[k];
  }
}

// Register-blocked FMA chains along y or z for both scales (lane x: taps ka/radius ra,
// lane y: taps kb/radius rb).  Same rotating-window scheme as the box sums.
template <class LoadF>
__device__ __forceinline__ void conv_chain(int c0, const float *ka, int ra, const float *kb, int rb,
                                           LoadF load, float2 (&acc)[kConvK]) {
  const int rm = max(ra, rb), L = 2 * rm + 1;
  float2 win[kConvK];
#pragma unroll
  for (int k = 0; k < kConvK; k++) { win[k] = load(c0 - rm + k); acc[k] = make_float2(0.f, 0.f); }
  for (int jb = 0; jb < L; jb += kConvK) {
#pragma unroll
    for (int u = 0; u < kConvK; u++) {
      const int j = jb + u;
      if (j < L) {
        const int jj = j - rm;
        const bool aa = jj >= -ra && jj <= ra, ab = jj >= -rb && jj <= rb;
        if (aa && ab) {
          const float2 kk = make_float2(ka[ra - jj], kb[rb - jj]);
#pragma unroll
          for (int k = 0; k < kConvK; k++) acc[k] = fma2(kk, win[(u + k) % kConvK], acc[k]);
        } else if (ab) {
          const float kk = kb[rb - jj];
#pragma unroll
          for (int k = 0; k < kConvK; k++) acc[k].y = __fmaf_rn(kk, win[(u + k) % kConvK].y, acc[k].y);
        } else if (aa) {
          const float kk = ka[ra - jj];
#pragma unroll
          for (int k = 0; k < kConvK; k++) acc[k].x = __fmaf_rn(kk, win[(u + k) % kConvK].x, acc[k].x);
        }
        win[u] = load(c0 - rm + j + kConvK);
      }
    }
  }
}

// ---------------------------------------------------------------- y pass
__global__ void k_conv_y(const Sub *subs, const __grid_constant__ DogTaps T, const float2 *in, float2 *out) {
  const Sub S = subs[blockIdx.y];
  const int rows_per_blk = blockDim.y * kConvK;
  const int tx_n = (S.W + 31) / 32, ty_n = (S.H + rows_per_blk - 1) / rows_per_blk;
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)tx_n * ty_n * S.D) return;
  const int z = (int)(bid / ((int64_t)tx_n * ty_n));
  const int rem = (int)(bid % ((int64_t)tx_n * ty_n));
  const int x = (rem % tx_n) * 32 + threadIdx.x;
  const int y0 = (rem / tx_n) * rows_per_blk + threadIdx.y * kConvK;
  if (x >= S.W || y0 >= S.H) return;
  const int P = S.P, H = S.H;
  const float2 *col = in + S.pvox + (int64_t)z * P * H + x;
  float2 acc[kConvK];
  conv_chain(y0, T.k[0], T.r[0], T.k[2], T.r[2],
             [&](int y) { return (y >= 0 && y < H) ? col[(int64_t)y * P] : make_float2(0.f, 0.f); }, acc);
  float2 *o = out + S.pvox + (int64_t)z * P * H + x;
#pragma unroll
  for (int k = 0; k < kConvK; k++)
    if (y0 + k < H) o[(int64_t)(y0 + k) * P] = acc[k];
}

// ---------------------------------------------------------------- z pass + subtract
// NormalizeSubtract3DKernel (DoG3DFilter.cu:346-354): dog = (small - large) * normalizer.  A
// thread owns kConvK slices of one column (threadIdx.y picks which, so the chunks of a column share their
// overlapping inputs through L1), over the padded plane.  Four 683x517x32 substacks, radii 2 / 4:
// 170 -> 140 us against one thread per whole column.
__global__ void __launch_bounds__(128) k_conv_z_dog(const Sub *subs, const __grid_constant__ DogTaps T, const float2 *in,
                                                    float *dog) {
  const Sub S = subs[blockIdx.z];
  const int64_t plane = (int64_t)S.P * S.H;
  const int64_t p = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const int D = S.D, z0 = (blockIdx.y * blockDim.y + threadIdx.y) * kConvK;
  if (p >= plane || z0 >= D) return;
  const float2 *col = in + S.pvox + p;
  float *o = dog + S.pvox + p;
  float2 acc[kConvK];
  conv_chain(z0, T.k[1], T.r[1], T.k[3], T.r[3],
             [&](int z) { return (z >= 0 && z < D) ? col[z * plane] : make_float2(0.f, 0.f); }, acc);
#pragma unroll
  for (int k = 0; k < kConvK; k++)
    if (z0 + k < D) o[(z0 + k) * plane] = __fmul_rn(__fsub_rn(acc[k].x, acc[k].y), T.normalizer);
}

// ---------------------------------------------------------------- the passes at known reaches
// The same passes with the wider scale's radius R at compile time: every tap of a thread's outputs is
// unrolled and takes its coefficient as a constant-bank operand of a scalar FMA (an f32x2 FMA takes registers
// only: two moves per coefficient pair and one per duplicated input made the f32x2 loops above four times as
// long), and all of a thread's inputs are in registers before the first tap.  The narrower
// scale's radius stays a launch value: one uniform test per tap.  Taps come centred: [j + R] is tap j.
// Near HBM.  Four 683x517x32 substacks, radii 3 / 5 and 2 / 4: x 191 -> 108 us, y 171 -> 151, z 140 -> 99.
constexpr int kConvMaxR = 14;
struct ConvTaps {
  float a[2 * kConvMaxR + 1], b[2 * kConvMaxR + 1];
  int ra;
  float normalizer;
};

template <int R>
__global__ void __launch_bounds__(32 * kConvXWarps) k_conv_x_t(const Sub *subs, const __grid_constant__ ConvTaps T,
                                                               const float *in, float2 *out) {
  constexpr int HX = (R + 3) / 4 * 4, NV = (HX + R + 4 + 3) / 4 * 4;   // inputs of a lane's four outputs, from 16 bytes on
  __shared__ __align__(16) float rows_sh[kConvXWarps][kConvXOut + 2 * HX + 4];
  const Sub S = subs[blockIdx.y];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, W = S.W, P = S.P;
  const int segs = (W + kConvXOut - 1) / kConvXOut;
  const int64_t id = (int64_t)blockIdx.x * kConvXWarps + w;
  if (id >= (int64_t)S.H * S.D * segs) return;
  const int64_t row = id / segs;
  const int x0 = (int)(id % segs) * kConvXOut;
  float *sh = rows_sh[w];
  const float *line = in + S.pvox + row * P;
#pragma unroll
  for (int i0 = 0; i0 < kConvXOut + 2 * HX + 4; i0 += 32) {
    const int i = i0 + lane, x = x0 - HX + i;
    if (i < kConvXOut + 2 * HX + 4) sh[i] = (x >= 0 && x < W) ? __ldg(line + x) : 0.0f;
  }
  __syncwarp();
  const int x = x0 + 4 * lane;
  if (x >= W) return;
  float v[NV];
#pragma unroll
  for (int i = 0; i < NV; i += 4) {
    const float4 f = *reinterpret_cast<const float4 *>(sh + 4 * lane + i);
    v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
  }
  float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int j = -R; j <= R; j++) {
    if ((j < 0 ? -j : j) <= T.ra)
#pragma unroll
      for (int o = 0; o < 4; o++) a[o] = __fmaf_rn(T.a[j + R], v[HX + j + o], a[o]);
#pragma unroll
    for (int o = 0; o < 4; o++) b[o] = __fmaf_rn(T.b[j + R], v[HX + j + o], b[o]);
  }
  float2 *o = out + S.pvox + row * P + x;
  if ((P & 3) == 0) {   // whole 32-byte sectors; columns past the width are padding
    float4 *o4 = reinterpret_cast<float4 *>(o);
    o4[0] = make_float4(a[0], b[0], a[1], b[1]);
    o4[1] = make_float4(a[2], b[2], a[3], b[3]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (x + k < W) o[k] = make_float2(a[k], b[k]);
  }
}

// kConvK outputs of a line from its kConvK + 2 R inputs v
template <int R>
__device__ __forceinline__ void conv_line(const ConvTaps &T, const float2 (&v)[kConvK + 2 * R], float (&a)[kConvK],
                                          float (&b)[kConvK]) {
#pragma unroll
  for (int k = 0; k < kConvK; k++) a[k] = b[k] = 0.0f;
#pragma unroll
  for (int j = -R; j <= R; j++) {
    if ((j < 0 ? -j : j) <= T.ra)
#pragma unroll
      for (int k = 0; k < kConvK; k++) a[k] = __fmaf_rn(T.a[j + R], v[k + j + R].x, a[k]);
#pragma unroll
    for (int k = 0; k < kConvK; k++) b[k] = __fmaf_rn(T.b[j + R], v[k + j + R].y, b[k]);
  }
}

template <int R>
__global__ void __launch_bounds__(128) k_conv_y_t(const Sub *subs, const __grid_constant__ ConvTaps T, const float2 *in,
                                                  float2 *out) {
  const Sub S = subs[blockIdx.y];
  const int rows_per_blk = blockDim.y * kConvK, P = S.P, H = S.H;
  const int tx_n = (S.W + 31) / 32, ty_n = (H + rows_per_blk - 1) / rows_per_blk;
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)tx_n * ty_n * S.D) return;
  const int z = (int)(bid / ((int64_t)tx_n * ty_n)), rem = (int)(bid % ((int64_t)tx_n * ty_n));
  const int x = (rem % tx_n) * 32 + threadIdx.x, y0 = (rem / tx_n) * rows_per_blk + threadIdx.y * kConvK;
  if (x >= S.W || y0 >= H) return;
  const int64_t base = S.pvox + (int64_t)z * P * H + x;
  float2 v[kConvK + 2 * R];
#pragma unroll
  for (int i = 0; i < kConvK + 2 * R; i++) {
    const int y = y0 - R + i;
    v[i] = y >= 0 && y < H ? __ldg(in + base + (int64_t)y * P) : make_float2(0.f, 0.f);
  }
  float a[kConvK], b[kConvK];
  conv_line<R>(T, v, a, b);
#pragma unroll
  for (int k = 0; k < kConvK; k++)
    if (y0 + k < H) out[base + (int64_t)(y0 + k) * P] = make_float2(a[k], b[k]);
}

template <int R>
__global__ void __launch_bounds__(128) k_conv_z_dog_t(const Sub *subs, const __grid_constant__ ConvTaps T, const float2 *in,
                                                      float *dog) {
  const Sub S = subs[blockIdx.z];
  const int64_t plane = (int64_t)S.P * S.H, p = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const int D = S.D, z0 = (blockIdx.y * blockDim.y + threadIdx.y) * kConvK;
  if (p >= plane || z0 >= D) return;
  float2 v[kConvK + 2 * R];
#pragma unroll
  for (int i = 0; i < kConvK + 2 * R; i++) {
    const int z = z0 - R + i;
    v[i] = z >= 0 && z < D ? __ldg(in + S.pvox + p + z * plane) : make_float2(0.f, 0.f);
  }
  float a[kConvK], b[kConvK];
  conv_line<R>(T, v, a, b);
  float *o = dog + S.pvox + p;
#pragma unroll
  for (int k = 0; k < kConvK; k++)
    if (z0 + k < D) o[(z0 + k) * plane] = __fmul_rn(__fsub_rn(a[k], b[k]), T.normalizer);
}

// ---------------------------------------------------------------- Hessian + PD mask
// The stage call's form, with the six planes.  A block stages its DoG tile and each thread forms the second differences
// of a column from it, the first derivatives along z in registers: 13 reads a voxel, where planes of first derivatives beside the tile cost 61 KB of shared memory
// (three blocks per SM), a second barrier and as many reads.  640x720x32 with planes: 200 -> 96 us, its 29 bytes a voxel
// 64.
// HZ: slices of a block, 16, or 8 where 16 leave SMs without one (a block works through its slices one after the other).
constexpr int kHX = 32, kHY = 8;                   // outputs per block and slice
constexpr int kDX = kHX + 8, kDY = kHY + 4;        // dog tile (halo 2, whole quads along x)

template <int HZ>
__global__ void __launch_bounds__(256) k_hessian_pd(const Sub *subs, const float *dog, uint8_t *mask,
                                                    float *hess6) {
  constexpr int kDZ = HZ + 4;
  __shared__ __align__(16) float sd[kDZ * kDY * kDX];
  const Sub S = subs[blockIdx.y];
  const int nx = (S.W + kHX - 1) / kHX, ny = (S.H + kHY - 1) / kHY, nz = (S.D + HZ - 1) / HZ;
  const int64_t bid = blockIdx.x;
  if (bid >= (int64_t)nx * ny * nz) return;
  const int bx = (int)(bid % nx), by = (int)((bid / nx) % ny), bz = (int)(bid / ((int64_t)nx * ny));
  const int x0 = bx * kHX, y0 = by * kHY, z0 = bz * HZ;
  const int W = S.W, H = S.H, D = S.D;
  const int64_t plane = (int64_t)W * H, pplane = (int64_t)S.P * H;
  const int lx = threadIdx.x, ly = threadIdx.y;
  if (W % 4 == 0 && (reinterpret_cast<uintptr_t>(dog + S.pvox) & 15) == 0) {   // quads lie inside or outside as a whole
    constexpr int kQ = kDX / 4;
    for (int i = ly * 32 + lx; i < kDZ * kDY * kQ; i += 256) {
      const int row = i / kQ, x = x0 - 4 + 4 * (i % kQ), y = y0 - 2 + row % kDY, z = z0 - 2 + row / kDY;
      reinterpret_cast<float4 *>(sd)[i] =
          y >= 0 && y < H && z >= 0 && z < D && x >= 0 && x < W
              ? __ldg(reinterpret_cast<const float4 *>(dog + S.pvox + z * pplane + (int64_t)y * S.P + x))
              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  } else {
#pragma unroll 8
    for (int i = ly * 32 + lx; i < kDZ * kDY * kDX; i += 256) {
      const int row = i / kDX, x = x0 - 4 + i % kDX, y = y0 - 2 + row % kDY, z = z0 - 2 + row / kDY;
      const bool in = y >= 0 && y < H && z >= 0 && z < D && x >= 0 && x < W;
      sd[i] = in ? __ldg(dog + S.pvox + z * pplane + (int64_t)y * S.P + x) : 0.0f;
    }
  }
  __syncthreads();
  const int x = x0 + lx, y = y0 + ly;
  if (x >= W || y >= H) return;
  // the tile holds zeros outside the volume; a first derivative there is zero too
  const bool xm = x >= 1, xp = x + 1 < W, ym = y >= 1, yp = y + 1 < H;
  constexpr int sy = kDX, sz = kDX * kDY;
  const int64_t nvox = plane * D;
  const float *c = sd + 2 * sz + (ly + 2) * sy + lx + 4;   // slice z0
  auto slice_x = [&](const float *q, bool in) { return in ? cdiff(q[1], q[-1]) : 0.0f; };
  auto slice_y = [&](const float *q, bool in) { return in ? cdiff(q[sy], q[-sy]) : 0.0f; };
  // first derivatives of slices z - 1 and z, the column's DoG of z and z + 1
  float gxm = slice_x(c - sz, z0 >= 1), gx0 = slice_x(c, true), gym = slice_y(c - sz, z0 >= 1), gy0 = slice_y(c, true);
  float gzm = z0 >= 1 ? cdiff(c[0], c[-2 * sz]) : 0.0f, gz0 = cdiff(c[sz], c[-sz]), c0 = c[0], c1 = c[sz];
  for (int lz = 0; lz < HZ && z0 + lz < D; lz++, c += sz) {
    const int z = z0 + lz;
    const bool zp = z + 1 < D;
    const float c2 = c[2 * sz], gxp = slice_x(c + sz, zp), gyp = slice_y(c + sz, zp), gzp = zp ? cdiff(c2, c0) : 0.0f;
    const float hxx = cdiff(xp ? cdiff(c[2], c0) : 0.0f, xm ? cdiff(c0, c[-2]) : 0.0f);
    const float hxy = cdiff(yp ? cdiff(c[sy + 1], c[sy - 1]) : 0.0f, ym ? cdiff(c[1 - sy], c[-1 - sy]) : 0.0f);
    const float hyy = cdiff(yp ? cdiff(c[2 * sy], c0) : 0.0f, ym ? cdiff(c0, c[-2 * sy]) : 0.0f);
    const float hxz = cdiff(gxp, gxm), hyz = cdiff(gyp, gym), hzz = cdiff(gzp, gzm);
    gxm = gx0; gx0 = gxp; gym = gy0; gy0 = gyp; gzm = gz0; gz0 = gzp; c0 = c1; c1 = c2;
    const int64_t i = z * plane + (int64_t)y * W + x;
    mask[S.vox + i] = pd_test(hxx, hxy, hxz, hyy, hyz, hzz) ? 1 : 0;
    if (hess6) {
      float *hp = hess6 + 6 * S.vox + i;
      hp[0] = hxx; hp[nvox] = hxy; hp[2 * nvox] = hxz;
      hp[3 * nvox] = hyy; hp[4 * nvox] = hyz; hp[5 * nvox] = hzz;
    }
  }
}

// ---------------------------------------------------------------- launchers
void launch_dog(const Sub *d_subs, int nsub, int max_w, int pitch, int max_h, int max_d, int64_t max_rows,
                const DogTaps &T, const float *norm, float2 *t0, float2 *t1, float *dog, cudaStream_t s) {
  // the unrolled passes where the large scale is the wider one and its radius is among the instantiations
  const int rx = T.r[2], rz = T.r[3], by = 4;
  ConvTaps C;
  auto centre = [&](int ka, int kb, int ra, int rb) {
    memset(&C, 0, sizeof(C));
    for (int j = -rb; j <= rb; j++) {
      if (j >= -ra && j <= ra) C.a[j + rb] = T.k[ka][ra - j];
      C.b[j + rb] = T.k[kb][rb - j];
    }
    C.ra = ra;
    C.normalizer = T.normalizer;
  };
  const dim3 gx(ceil_div(max_rows * ceil_div(max_w, kConvXOut), kConvXWarps), nsub);
  const dim3 gy((unsigned)((int64_t)ceil_div(max_w, 32) * ceil_div(max_h, by * kConvK) * max_d), nsub);
  const dim3 gz(ceil_div((int64_t)pitch * max_h, 32), ceil_div(max_d, by * kConvK), nsub);
  bool done = false;
  if (T.r[0] <= rx && rx >= 2 && rx <= kConvMaxR) {
    centre(0, 2, T.r[0], rx);
    done = true;
    switch (rx) {
#define HDOG_CASE(R)                                                                                             \
  case R:                                                                                                        \
    KLAUNCH("k_conv_x", s, (k_conv_x_t<R><<<gx, 32 * kConvXWarps, 0, s>>>(d_subs, C, norm, t0)));                \
    KLAUNCH("k_conv_y", s, (k_conv_y_t<R><<<gy, dim3(32, by), 0, s>>>(d_subs, C, t0, t1)));                      \
    break;
      HDOG_CASE(2) HDOG_CASE(3) HDOG_CASE(4) HDOG_CASE(5) HDOG_CASE(6) HDOG_CASE(7) HDOG_CASE(8) HDOG_CASE(9)
      HDOG_CASE(10) HDOG_CASE(11) HDOG_CASE(12) HDOG_CASE(13) HDOG_CASE(14)
#undef HDOG_CASE
    }
  }
  if (!done) {
    KLAUNCH("k_conv_x", s, (k_conv_x<<<gx, 32 * kConvXWarps, 0, s>>>(d_subs, T, norm, t0)));
    KLAUNCH("k_conv_y", s, (k_conv_y<<<gy, dim3(32, by), 0, s>>>(d_subs, T, t0, t1)));
  }
  if (T.r[1] <= rz && rz >= 2 && rz <= 8) {
    centre(1, 3, T.r[1], rz);
    switch (rz) {
#define HDOG_CASE(R)                                                                                             \
  case R:                                                                                                        \
    KLAUNCH("k_conv_z_dog", s, (k_conv_z_dog_t<R><<<gz, dim3(32, by), 0, s>>>(d_subs, C, t1, dog)));             \
    return;
      HDOG_CASE(2) HDOG_CASE(3) HDOG_CASE(4) HDOG_CASE(5) HDOG_CASE(6) HDOG_CASE(7) HDOG_CASE(8)
#undef HDOG_CASE
    }
  }
  KLAUNCH("k_conv_z_dog", s, (k_conv_z_dog<<<gz, dim3(32, by), 0, s>>>(d_subs, T, t1, dog)));
}

void launch_hessian_pd(const Sub *d_subs, int nsub, int max_w, int max_h, int max_d, const float *dog,
                       uint8_t *mask, float *hess6, cudaStream_t s) {
  const int64_t cols = (int64_t)ceil_div(max_w, kHX) * ceil_div(max_h, kHY);
  const int hz = cols * ceil_div(max_d, 16) * nsub >= 152 ? 16 : 8;
  const dim3 grid((unsigned)(cols * ceil_div(max_d, hz)), nsub);
  KLAUNCH("k_hessian_pd", s, ((hz == 16 ? k_hessian_pd<16> : k_hessian_pd<8>)<<<grid, dim3(kHX, kHY), 0, s>>>(d_subs, dog, mask, hess6)));
}

}  // namespace hdog
