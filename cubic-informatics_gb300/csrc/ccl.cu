// ccl.cu -- 3D connected-component labelling with the reference's connectivity, sm_103a.
//
// Reference: src/3D/CCL3D.cu (CCL :81-117).  The reference iterates neighbour-min scans
// and pointer jumping, synchronising with the host twice per iteration.  Its fixed point
// labels each component with the minimum linear index of its voxels, over a graph whose
// edges are the 26 LINEAR offsets dz*W*H + dy*W + dx kept inside [0, N) -- so a row end
// touches the next row's start and a slice's last row the next slice's first -- and in
// which voxel 0 is background (label = index * mask).
//
// Here the same labels come from union-find in three passes, with no host round trip:
//   1. k_ccl_local: a 64 x 16 tile of 32 slices (16 or 8 in small batches) is labelled in
//      shared memory over its 2 x 2 x 2 cells (see below); the foreground edges that
//      leave the tile (its faces, and the wrap-around offsets) go to an edge list.
//   2. k_ccl_edges: a persistent pass merges those edges in the global label array.
//      If the list overflowed, k_ccl_cross_direct merges the same edges from the mask.
//   3. k_ccl_flatten: every foreground voxel gets its root (a read-only walk, so every
//      store is final); roots are recorded in a bitmap and counted per 4096 voxels for
//      the region numbering.
// Linking always hangs the larger root under the smaller, so roots are component minima.
#include "kernels.cuh"

namespace hdog {

// ------------------------------------------------------------------ global union-find
// Invariants: a parent pointer only ever points to a smaller index in the same tree; a
// root is linked only by a compare-and-swap that requires it to still be a root, so
// trees merge but never split.  A stale read (the L1 cache is not coherent across SMs)
// can then only show an older pointer of the same tree: two finds that meet at one node
// are truly in one tree, and a link attempted on a former root fails and retries from
// its current parent.  Path halving stores only an ancestor of the node's parent.
__device__ __forceinline__ int32_t uf_find(int32_t *L, int32_t a, int64_t limit, int *status) {
  int32_t p = __ldcg(L + a);
  int64_t steps = 0;
  while (p != a) {
    const int32_t gp = __ldcg(L + p);
    if (gp != p) L[a] = gp;
    a = p;
    p = gp;
    if (++steps > limit) { atomicExch(status, HDOG_ERR_TIMEOUT); break; }
  }
  return a;
}

// Read-only walk, for the flatten pass where every store must be a final root.
__device__ __forceinline__ int32_t uf_root(const int32_t *L, int32_t a, int64_t limit, int *status) {
  int32_t p = __ldcg(L + a);
  int64_t steps = 0;
  while (p != a) {
    a = p;
    p = __ldcg(L + a);
    if (++steps > limit) { atomicExch(status, HDOG_ERR_TIMEOUT); break; }
  }
  return a;
}

__device__ __forceinline__ void uf_union(int32_t *L, int32_t a, int32_t b, int64_t limit, int *status) {
  for (int64_t it = 0; it <= limit; it++) {
    a = uf_find(L, a, limit, status);
    b = uf_find(L, b, limit, status);
    if (a == b) return;
    if (a > b) { const int32_t t = a; a = b; b = t; }
    const int32_t cur = atomicCAS(&L[b], b, a);
    if (cur == b) return;
    b = cur;
  }
  atomicExch(status, HDOG_ERR_TIMEOUT);
}

// The 13 backward linear offsets (the other 13 of the 26 are their mirror images).
__device__ __forceinline__ void back_offset(int k, int &dz, int &dy, int &dx) {
  dz = k < 9 ? -1 : 0;
  dy = k < 9 ? k / 3 - 1 : (k < 12 ? -1 : 0);
  dx = k < 9 ? k % 3 - 1 : (k < 12 ? k - 10 : -1);
}

// ------------------------------------------------------------------ pass 1: tile-local
// Tiles of 64 x 16 voxels and TZ slices.  A block works through its tile's layers one after the other, so
// where the 32-slice tiles would leave most of the chip idle (fewer than two per SM) they are 16 slices
// deep, and 8 where even those are fewer than one for two SMs: more cross-tile edges, but shorter blocks and
// more of them.  One 128x96x16 substack 27 -> 16 us, one of 256x256x32 50 -> 31 us
// (13.6 and 24.6 with the cells' tests packed as below).
constexpr int kTX = 64, kTY = 16;
constexpr int kCclThreads = 256;              // thread = 4 x-consecutive voxels of one row, all TZ slices

// Shared-memory union-find over the tile's cells, 32-bit parents (native shared atomics;
// kBg32 marks a background cell).  Find with path halving (stores an ancestor of the
// parent only, as in the global version); without it "smaller root wins" linking grows
// long chains.
constexpr uint32_t kBg32 = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t sfind(volatile uint32_t *par, uint32_t t) {
  uint32_t p = par[t];
  while (p != t) {
    const uint32_t gp = par[p];
    if (gp != p) par[t] = gp;
    t = p;
    p = gp;
  }
  return t;
}

// Read-only find for the final pass over a finished forest.
__device__ __forceinline__ uint32_t sroot(const uint32_t *par, uint32_t t) {
  uint32_t p = par[t];
  while (p != t) {
    t = p;
    p = par[t];
  }
  return t;
}

__device__ __forceinline__ void sunion(uint32_t *par, uint32_t a, uint32_t b, uint32_t limit) {
  volatile uint32_t *v = par;
  for (uint32_t it = 0; it < limit; it++) {
    a = sfind(v, a);
    b = sfind(v, b);
    if (a == b) return;
    if (a > b) { const uint32_t t = a; a = b; b = t; }
    const uint32_t cur = atomicCAS(&par[b], b, a);
    if (cur == b) return;
    b = cur;
  }
}

struct CclTile {
  int x0, y0, z0, tz;     // origin, slices in this tile
};

template <int TZ>
__device__ __forceinline__ bool ccl_tile(const Sub &S, int64_t bid, CclTile &T) {
  const int nx = (S.W + kTX - 1) / kTX, ny = (S.H + kTY - 1) / kTY, nz = (S.D + TZ - 1) / TZ;
  if (bid >= (int64_t)nx * ny * nz) return false;
  T.x0 = (int)(bid % nx) * kTX;
  T.y0 = (int)((bid / nx) % ny) * kTY;
  T.z0 = (int)(bid / ((int64_t)nx * ny)) * TZ;
  T.tz = min(TZ, S.D - T.z0);
  return true;
}

// Backward neighbour (dz, dy, dx) of voxel (x, y, z), tile coordinates (lx, ly, lz):
// true when the edge is not a plain 3D step inside this tile (it leaves the tile, or
// it wraps around a row or slice end).
__device__ __forceinline__ bool leaves_tile(const Sub &S, const CclTile &T, int x, int y, int z, int lx, int ly,
                                            int lz, int dz, int dy, int dx) {
  const int nx = x + dx, ny = y + dy, nz = z + dz;
  const bool in_vol = nx >= 0 && nx < S.W && ny >= 0 && ny < S.H && nz >= 0;
  const bool in_tile = lx + dx >= 0 && lx + dx < kTX && ly + dy >= 0 && ly + dy < kTY && lz + dz >= 0 && lz + dz < T.tz;
  return !(in_vol && in_tile);
}

constexpr int kEdgeBuf = 2048;                // cross-tile edges staged per tile before one global reservation

// ---- cell union-find inside the tile
// Inside a tile every edge is a plain 26-neighbour step (the reference's row and slice
// wrap-arounds always leave the tile and go to the edge list), and any two foreground
// voxels of one 2 x 2 x 2 cell are 26-neighbours.  So the tile is labelled over cells:
// a cell is one union-find node, its 8-bit occupancy says which voxels are foreground
// (bit 4*dz + 2*dy + dx, i.e. linear voxel order), and two neighbouring cells are
// connected exactly when each has a foreground voxel on the side facing the other --
// two mask tests per pair.  A component's label is then the minimum voxel index over
// its cells, found with one shared-memory atomicMin per cell.
constexpr int kCX = kTX / 2, kCY = kTY / 2;

// Occupancy bits of a cell whose voxels have local coordinate `side` along one axis
// (0 or 1); axis 0 = x, 1 = y, 2 = z.
__host__ __device__ constexpr uint8_t cell_side(int axis, int side) {
  uint8_t m = 0;
  for (int v = 0; v < 8; v++)
    if (((v >> axis) & 1) == side) m |= (uint8_t)(1u << v);
  return m;
}
// For cell offset d (-1, 0, +1) along an axis: the voxels of this cell (self) and of the
// neighbour that can touch across it.
__host__ __device__ constexpr uint8_t cell_face(int axis, int d, bool self) {
  return d == 0 ? (uint8_t)0xFF : (d < 0 ? cell_side(axis, self ? 0 : 1) : cell_side(axis, self ? 1 : 0));
}
struct CellNb {
  int dz, dy, dx;
  uint8_t self, other;
};
__host__ __device__ constexpr CellNb cell_nb(int dz, int dy, int dx) {
  return CellNb{dz, dy, dx,
                (uint8_t)(cell_face(0, dx, true) & cell_face(1, dy, true) & cell_face(2, dz, true)),
                (uint8_t)(cell_face(0, dx, false) & cell_face(1, dy, false) & cell_face(2, dz, false))};
}
// The 13 backward cell neighbours (the other 13 are their mirror images) as four words of occupancy bytes: the layer
// below at dx = -1, 0, +1, each with dy = -1, 0, +1 in bytes 0 .. 2, and this layer's (dy, dx) = (-1, -1), (-1, 0),
// (-1, +1), (0, -1).  A link list has bit 8 b + w for byte b of word w, so a word's tests are a few operations on all its
// bytes at once instead of two masks and two branches a neighbour.  The kernel is bound by its ALU
// instructions, of which these tests and the cells' occupancy were the most: 1.42 G voxels 4.07 -> 2.91 ms with both packed,
// a row's eight cells stored at once and a column's neighbours read from the next lanes.
struct CellWords {
  uint32_t w[4];
};
__host__ __device__ constexpr CellNb word_nb(int w, int b) {
  return w < 3 ? cell_nb(-1, b - 1, w - 1) : (b < 3 ? cell_nb(0, -1, b - 1) : cell_nb(0, 0, -1));
}
// self / other masks of a word's bytes; flat: the cells as neighbours of the one below instead (dz = 0)
__host__ __device__ constexpr uint32_t word_mask(int w, bool self, bool flat) {
  uint32_t m = 0;
  for (int b = 0; b < (w < 3 ? 3 : 4); b++) {
    const CellNb n = flat ? cell_nb(0, b - 1, w - 1) : word_nb(w, b);
    m |= (uint32_t)(self ? n.self : n.other) << (8 * b);
  }
  return m;
}
// 0x80 in every nonzero byte
__device__ __forceinline__ uint32_t byte_flags(uint32_t x) {
  return (((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u;
}
// Link list of a cell with occupancy oc.
__device__ __forceinline__ uint32_t cell_links(uint32_t oc, const CellWords &n) {
  constexpr uint32_t own[4] = {word_mask(0, true, false), word_mask(1, true, false), word_mask(2, true, false), word_mask(3, true, false)};
  constexpr uint32_t nbr[4] = {word_mask(0, false, false), word_mask(1, false, false), word_mask(2, false, false), word_mask(3, false, false)};
  const uint32_t r = oc * 0x01010101u;
  uint32_t todo = 0;
#pragma unroll
  for (int w = 0; w < 4; w++) todo |= (byte_flags(r & own[w]) & byte_flags(n.w[w] & nbr[w])) >> (7 - w);
  return todo;
}
constexpr uint32_t kLinkBelow = 1u << 9, kLinkBehind = 1u << 11, kLinkLeft = 1u << 27;   // (-1,0,0), (0,-1,0), (0,0,-1)
// Links to the layer below whose cell the cell directly below touches in that layer.
__device__ __forceinline__ uint32_t below_touches(const CellWords &n) {
  constexpr uint32_t own[3] = {word_mask(0, true, true), word_mask(1, true, true), word_mask(2, true, true)};
  constexpr uint32_t nbr[3] = {word_mask(0, false, true), word_mask(1, false, true), word_mask(2, false, true)};
  const uint32_t r = ((n.w[1] >> 8) & 0xFFu) * 0x01010101u;
  uint32_t t = 0;
#pragma unroll
  for (int w = 0; w < 3; w++) t |= (byte_flags(r & own[w]) & byte_flags(n.w[w] & nbr[w])) >> (7 - w);
  return t & ~kLinkBelow;
}
// Cell offset of list bit p.
__device__ __forceinline__ void link_offset(int p, int &dz, int &dy, int &dx) {
  const int w = p & 7, b = p >> 3;
  dz = w < 3 ? -1 : 0;
  dy = w < 3 ? b - 1 : (b < 3 ? -1 : 0);
  dx = w < 3 ? w - 1 : (b < 3 ? b - 1 : -1);
}

// Occupancy of a halo-framed block of cells: the tile's cells plus one cell on each x
// and y side and one layer below (cell coordinates -1 .. kC? along each axis).
// Rows of 40 bytes with cell 0 at byte 8: eight cells of a row are one 8-byte store.
constexpr int kHX = kCX + 8, kHY = kCY + 2;
__device__ __forceinline__ int halo_of(int cx, int cy, int cz) { return ((cz + 1) * kHY + (cy + 1)) * kHX + (cx + 8); }
__device__ __forceinline__ int cell_bit(int lx, int ly, int lz) { return ((lz & 1) << 2) | ((ly & 1) << 1) | (lx & 1); }

// Occupancy of the cell whose first voxel is (x, y, z) (volume coordinates; voxels outside
// the volume, past depth_valid handling or at index 0 count as background).
__device__ __forceinline__ uint32_t cell_occ(const Sub &S, const uint8_t *m, int64_t WH, int x, int y, int z) {
  uint32_t o = 0;
  if (x + 1 < 0 || x >= S.W || y + 1 < 0 || y >= S.H || z + 1 < 0 || z >= S.D) return 0;
  // both voxels in one load: x is even, so a caller's mask on an even address and an even width put them on two bytes
  const bool pair = x >= 0 && x + 1 < S.W && S.W % 2 == 0 && (reinterpret_cast<uintptr_t>(m) & 1u) == 0;
#pragma unroll
  for (int dz = 0; dz < 2; dz++)
#pragma unroll
    for (int dy = 0; dy < 2; dy++) {
      const int zz = z + dz, yy = y + dy;
      if (zz < 0 || zz >= S.D || yy < 0 || yy >= S.H) continue;
      const int64_t g = zz * WH + (int64_t)yy * S.W + x;
      uint32_t v;
      if (pair) {
        const uint16_t two = __ldg(reinterpret_cast<const uint16_t *>(m + g));
        v = ((two & 0xFFu) ? 1u : 0u) | ((two >> 8) ? 2u : 0u);
      } else {
        v = (x >= 0 && m[g]) ? 1u : 0u;
        if (x + 1 < S.W && m[g + 1]) v |= 2u;
      }
      if (g == 0) v &= ~1u;   // voxel 0 is background
      o |= v << (4 * dz + 2 * dy);
    }
  return o;
}

// Occupancy bytes of the 8 cells whose first voxels are (x + 2k, y, z), k = 0..7, from one
// 16-byte load of each of the 4 voxel rows they cover (x 16-byte aligned, x + 15 < W;
// rows outside the volume read as background).
__device__ __forceinline__ uint2 cell_occ8(const Sub &S, const uint8_t *m, int64_t WH, int x, int y, int z) {
  uint4 r[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int zz = z + (q >> 1), yy = y + (q & 1);
    r[q] = (zz >= 0 && zz < S.D && yy >= 0 && yy < S.H)
               ? __ldg(reinterpret_cast<const uint4 *>(m + zz * WH + (int64_t)yy * S.W + x))
               : make_uint4(0u, 0u, 0u, 0u);
  }
  uint32_t o[4] = {0u, 0u, 0u, 0u};   // cells 2j and 2j + 1 in bytes 0 and 2
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int sh = 4 * (q >> 1) + 2 * (q & 1);   // bit of the row's first voxel: 4 dz + 2 dy
    const uint32_t w[4] = {r[q].x, r[q].y, r[q].z, r[q].w};
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t f = byte_flags(w[j]);   // voxels 0, 1 at bits 7, 15 and 2, 3 at 23, 31
      o[j] |= (((f >> 7) | (f >> 14)) & 0x00030003u) << sh;
    }
  }
  return make_uint2(__byte_perm(o[0], o[1], 0x6420), __byte_perm(o[2], o[3], 0x6420));
}

// Drops links that other links of the tile already imply.  Every tile edge is linked by
// the later of its two cells, so with cell c linked to B (a backward neighbour) and B
// touching A (another backward neighbour of c), the edge B-A is linked too and c-A adds
// nothing.  Links kept unconditionally: below (dz -1), behind (dy -1), left (dx -1).  Pruned:
//   via below:   the other eight cells of the layer below, through the
//                in-plane edges of that layer;
//   via behind:  its left and right neighbours through that row's x edges (kept by rule) and
//                the cell below it through its own link below (kept);
//   via left:    the cell behind it and the one below it through its links (both kept).
// Each pruned link rests on links that are kept or pruned only by the rules for
// in-layer edges, which rest on kept links: the implied connectivity is exact.
// The component minima are unchanged (they come from the final trees, not the links).
__device__ __forceinline__ bool touches(uint32_t a, uint32_t b, CellNb e) { return (a & e.self) && (b & e.other); }

__device__ __forceinline__ uint32_t prune_links(uint32_t todo, const CellWords &n) {
  if (todo & kLinkBelow) todo &= ~below_touches(n);
  if (todo & kLinkBehind) {
    const uint32_t on10 = (n.w[3] >> 8) & 0xFFu;
    if (touches(on10, n.w[3] & 0xFFu, cell_nb(0, 0, -1))) todo &= ~(1u << 3);
    if (touches(on10, (n.w[3] >> 16) & 0xFFu, cell_nb(0, 0, 1))) todo &= ~(1u << 19);
    if (touches(on10, n.w[1] & 0xFFu, cell_nb(-1, 0, 0))) todo &= ~(1u << 1);
  }
  if (todo & kLinkLeft) {
    const uint32_t on12 = n.w[3] >> 24;
    if (touches(on12, n.w[3] & 0xFFu, cell_nb(0, -1, 0))) todo &= ~(1u << 3);
    if (touches(on12, (n.w[0] >> 8) & 0xFFu, cell_nb(-1, 0, 0))) todo &= ~(1u << 8);
  }
  return todo;
}

template <int TZ>
__global__ void __launch_bounds__(kCclThreads, 4) k_ccl_local(const Sub *subs, const uint8_t *mask, int32_t *labels,
                                                          int2 *edges, unsigned long long *edge_count) {
  constexpr int kCZ = TZ / 2, kCells = kCX * kCY * kCZ, kHZ = kCZ + 1, kHalo = kHX * kHY * kHZ;   // 4096 cells, 6800 bytes with halo at TZ 32
  static_assert(kCX == 32, "a warp is a row of cells");
  __shared__ __align__(16) uint32_t par[kCells];
  __shared__ __align__(8) uint8_t occ[kHalo + 8];   // cell 32 of a row is byte 0 of the next
  __shared__ uint32_t minv[kCells];
  __shared__ int2 ebuf[kEdgeBuf];
  __shared__ uint32_t n_local_edges;
  __shared__ unsigned long long edge_base;
  const Sub S = subs[blockIdx.y];
  CclTile T;
  if (!ccl_tile<TZ>(S, blockIdx.x, T)) return;
  const int t = threadIdx.x;
  const int64_t WH = (int64_t)S.W * S.H;
  const int64_t N = WH * S.D;
  const uint8_t *m = mask + S.vox;
  if (t == 0) n_local_edges = 0;
  // 1. occupancy of the tile's cells and of the halo (the layer below only when the tile
  //    does not start at slice 0); union-find nodes for the tile's cells.  Rows of 16-byte
  //    aligned tiles inside the volume are read 16 voxels (8 cells) per load; the halo's
  //    side columns, and every cell of other tiles, one cell at a time.
  const int ncz = (T.tz + 1) / 2;
  const bool rows16 = S.W % 16 == 0 && T.x0 + kTX <= S.W && (reinterpret_cast<uintptr_t>(m) & 15u) == 0;
  if (rows16) {
    constexpr int kSeg = kCX / 8;   // 8-cell segments per cell row
    for (int it = t; it < kHY * kHZ * kSeg; it += kCclThreads) {
      const int seg = it % kSeg, hy = (it / kSeg) % kHY, hz = it / (kSeg * kHY);
      const int cy = hy - 1, cz = hz - 1, cx0 = seg * 8;
      uint2 o = make_uint2(0u, 0u);
      if (cz < ncz && (cz >= 0 || T.z0 > 0)) {
        o = cell_occ8(S, m, WH, T.x0 + 2 * cx0, T.y0 + 2 * cy, T.z0 + 2 * cz);
        if (T.x0 == 0 && T.y0 + 2 * cy == 0 && T.z0 + 2 * cz == 0 && cx0 == 0) o.x &= ~1u;   // voxel 0
        if (cz >= 0 && 2 * cz + 1 >= T.tz) { o.x &= 0x0F0F0F0Fu; o.y &= 0x0F0F0F0Fu; }
      }
      *reinterpret_cast<uint2 *>(occ + halo_of(cx0, cy, cz)) = o;
      if (cy >= 0 && cy < kCY && cz >= 0) {
        const uint32_t c = (cz * kCY + cy) * kCX + cx0;
        uint4 *pc = reinterpret_cast<uint4 *>(par + c);
        pc[0] = make_uint4(o.x & 0xFFu ? c : kBg32, o.x & 0xFF00u ? c + 1 : kBg32, o.x & 0xFF0000u ? c + 2 : kBg32, o.x >> 24 ? c + 3 : kBg32);
        pc[1] = make_uint4(o.y & 0xFFu ? c + 4 : kBg32, o.y & 0xFF00u ? c + 5 : kBg32, o.y & 0xFF0000u ? c + 6 : kBg32, o.y >> 24 ? c + 7 : kBg32);
      }
    }
  }
  for (int h = t; h < kHY * kHZ * (rows16 ? 2 : kCX + 2); h += kCclThreads) {
    int hx, hy, hz;
    if (rows16) {   // the side columns cx = -1 and cx = kCX
      hx = (h & 1) ? kCX + 1 : 0;
      hy = (h >> 1) % kHY;
      hz = (h >> 1) / kHY;
    } else {
      hx = h % (kCX + 2);
      hy = (h / (kCX + 2)) % kHY;
      hz = h / ((kCX + 2) * kHY);
    }
    const int cx = hx - 1, cy = hy - 1, cz = hz - 1;
    uint32_t o = 0;
    if (cz < ncz && (cz >= 0 || T.z0 > 0)) {
      o = cell_occ(S, m, WH, T.x0 + 2 * cx, T.y0 + 2 * cy, T.z0 + 2 * cz);
      if (cz >= 0 && 2 * cz + 1 >= T.tz) o &= 0x0Fu;   // a tile's last odd slice: no second layer
    }
    occ[halo_of(cx, cy, cz)] = (uint8_t)o;
    if (cx >= 0 && cx < kCX && cy >= 0 && cy < kCY && cz >= 0) {
      const int c = (cz * kCY + cy) * kCX + cx;
      par[c] = o ? (uint32_t)c : kBg32;
    }
  }
  __syncthreads();
  // 2. unions between neighbouring cells of the tile.  The unrolled neighbour tests only
  //    collect a 13-bit list per cell, parked in minv (unused until step 3); the unions then
  //    run in warp-wide rounds over the lane's whole cell column, one link per lane and
  //    round, re-converged after each, so lanes whose finds and retries differ in length do
  //    not split the warp, and a lane with many links in one layer does not hold the
  //    others idle for that layer alone.  Union order does not change the components.
  const int cx = t % kCX, cy = t / kCX;
  uint32_t layers = 0;   // bit cz: the cell of layer cz has links
  {
    // the column's cells of rows cy - 1 .. cy + 1 (0 outside the tile) in bytes 0 .. 2, its neighbours' by shuffles; a
    // layer's words stay in registers as the next one's layer below
    const uint32_t rows = (cy > 0 ? 0xFFu : 0u) | 0xFF00u | (cy < kCY - 1 ? 0xFF0000u : 0u);
    CellWords n = {{0u, 0u, 0u, 0u}};
    for (int cz = 0; cz < ncz; cz++) {
      const uint8_t *o = occ + halo_of(cx, cy - 1, cz);
      const uint32_t cur = (o[0] | (uint32_t)o[kHX] << 8 | (uint32_t)o[2 * kHX] << 16) & rows;
      uint32_t left = __shfl_up_sync(0xFFFFFFFFu, cur, 1), right = __shfl_down_sync(0xFFFFFFFFu, cur, 1);
      if (cx == 0) left = 0;
      if (cx == kCX - 1) right = 0;
      const uint32_t oc = (cur >> 8) & 0xFFu;
      uint32_t todo = 0;
      if (oc) {
        n.w[3] = __byte_perm(__byte_perm(left, cur, 0x1040), right, 0x3410);
        todo = prune_links(cell_links(oc, n), n);
      }
      minv[(cz * kCY + cy) * kCX + cx] = todo;
      layers |= (todo ? 1u : 0u) << cz;
      n.w[0] = left; n.w[1] = cur; n.w[2] = right;
    }
  }
  {
    uint32_t todo = 0;
    int c = 0;
    while (__any_sync(0xFFFFFFFFu, todo != 0 || layers != 0)) {
      if (!todo && layers) {
        const int cz = __ffs(layers) - 1;
        layers &= layers - 1;
        c = (cz * kCY + cy) * kCX + cx;
        todo = minv[c];
      }
      if (todo) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1;
        int dz, dy, dx;
        link_offset(k, dz, dy, dx);
        const int cn = c + (dz * kCY + dy) * kCX + dx;
        if (par[cn] != par[c]) sunion(par, c, cn, 2 * kCells);
      }
      __syncwarp();
    }
  }
  for (int cz = 0; cz < ncz; cz++) minv[(cz * kCY + cy) * kCX + cx] = 0xFFFFFFFFu;
  __syncthreads();
  // 3. roots in place, then each component's minimum voxel (tile order = volume order)
  for (int cz = 0; cz < ncz; cz++) {
    const int c = (cz * kCY + cy) * kCX + cx;
    if (occ[halo_of(cx, cy, cz)]) par[c] = sroot(par, c);
  }
  __syncthreads();
  for (int cz = 0; cz < ncz; cz++) {
    const int c = (cz * kCY + cy) * kCX + cx;
    const uint32_t oc = occ[halo_of(cx, cy, cz)];
    if (!oc) continue;
    const int b = __ffs(oc) - 1;   // first voxel of the cell in linear order
    const uint32_t v = ((2 * cz + (b >> 2)) * kTY + 2 * cy + ((b >> 1) & 1)) * kTX + 2 * cx + (b & 1);
    atomicMin(&minv[par[c]], v);
  }
  // 4a. plain cross-tile edges, cell to cell: a face cell and its backward neighbour cell
  //     outside the tile are connected when their facing voxels are foreground; the edge
  //     joins the first foreground voxel of each
  auto first_voxel = [&](int ccx, int ccy, int ccz, uint32_t o) -> int64_t {
    const int b = __ffs(o) - 1;
    return (int64_t)(T.z0 + 2 * ccz + (b >> 2)) * WH + (int64_t)(T.y0 + 2 * ccy + ((b >> 1) & 1)) * S.W + T.x0 +
           2 * ccx + (b & 1);
  };
  auto emit = [&](int64_t a, int64_t b) {
    const uint32_t i = atomicAdd(&n_local_edges, 1u);
    if (i < (uint32_t)kEdgeBuf) {
      ebuf[i] = make_int2((int32_t)a, (int32_t)b);
    } else {
      const unsigned long long j = atomicAdd(&edge_count[blockIdx.y], 1ull);
      if ((int64_t)j < S.edge_cap) edges[S.edge + j] = make_int2((int32_t)a, (int32_t)b);
    }
  };
  {
    constexpr int kFacePerLayer = 2 * kCX + 2 * (kCY - 2);   // rows cy = 0, kCY-1 and columns cx = 0, kCX-1
    const bool zface = T.z0 > 0;
    const int nf = zface ? ncz * kFacePerLayer + kCX * kCY : ncz * kFacePerLayer;
    for (int f = t; f < nf; f += kCclThreads) {
      int fx, fy, fz;
      if (f < ncz * kFacePerLayer) {
        fz = f / kFacePerLayer;
        const int j = f % kFacePerLayer;
        if (j < kCX) { fx = j; fy = 0; }
        else if (j < 2 * kCX) { fx = j - kCX; fy = kCY - 1; }
        else if (j < 2 * kCX + kCY - 2) { fx = 0; fy = j - 2 * kCX + 1; }
        else { fx = kCX - 1; fy = j - 2 * kCX - (kCY - 2) + 1; }
      } else {   // the bottom layer of a tile above slice 0, interior cells (faces done above)
        const int j = f - ncz * kFacePerLayer;
        fx = j % kCX; fy = j / kCX; fz = 0;
        if (fx == 0 || fx == kCX - 1 || fy == 0 || fy == kCY - 1) continue;
      }
      const uint32_t oc = occ[halo_of(fx, fy, fz)];
      if (!oc) continue;
      const uint8_t *o = occ + halo_of(fx, fy, fz), *below = o - kHX * kHY;
      CellWords n;
#pragma unroll
      for (int w = 0; w < 3; w++)
        n.w[w] = below[w - 1 - kHX] | (uint32_t)below[w - 1] << 8 | (uint32_t)below[w - 1 + kHX] << 16;
      n.w[3] = o[-1 - kHX] | (uint32_t)o[-kHX] << 8 | (uint32_t)o[1 - kHX] << 16 | (uint32_t)o[-1] << 24;
      // links to cells beyond the tile's x and y faces, and to the layer below it
      const uint32_t side = (fx == 0 ? 0x08010109u : 0u) | (fx == kCX - 1 ? 0x000C0404u : 0u) |
                            (fy == 0 ? 0x0008080Fu : 0u) | (fy == kCY - 1 ? 0x00070000u : 0u);
      uint32_t todo = cell_links(oc, n) & (side | (fz == 0 ? 0x00070707u : 0u));
      // linked to the cell below, in the tile below: that tile's own unions join it to those of its eight
      // neighbours it touches inside the same footprint, so the edges to these add nothing
      if (todo & kLinkBelow) todo &= ~(below_touches(n) & ~side);
      if (!todo) continue;
      const int64_t a = first_voxel(fx, fy, fz, oc);
      while (todo) {
        const int k = __ffs(todo) - 1;
        todo &= todo - 1;
        int dz, dy, dx;
        link_offset(k, dz, dy, dx);
        const int nx = fx + dx, ny = fy + dy, nz = fz + dz;
        emit(a, first_voxel(nx, ny, nz, occ[halo_of(nx, ny, nz)]));
      }
    }
  }
  // 4b. the reference's wrap-around edges: backward linear offsets of a voxel in the first
  //     or last column or row that leave the row or slice (only border tiles hold such voxels)
  if (T.x0 == 0 || T.x0 + kTX >= S.W || T.y0 == 0 || T.y0 + kTY >= S.H) {
    // per layer: the first and last column of the volume (all rows), then the first and last row
    constexpr int kRing = 2 * kTY + 2 * kTX;
    for (int v = t; v < kRing * T.tz; v += kCclThreads) {
      const int lz = v / kRing, j = v % kRing;
      int lx, ly;
      if (j < 2 * kTY) {
        lx = (j & 1 ? S.W - 1 : 0) - T.x0;
        ly = j >> 1;
      } else {
        ly = ((j & 1) ? S.H - 1 : 0) - T.y0;
        lx = (j - 2 * kTY) >> 1;
        if (T.x0 + lx == 0 || T.x0 + lx == S.W - 1) continue;   // done with the columns
      }
      const int x = T.x0 + lx, y = T.y0 + ly, z = T.z0 + lz;
      if (lx < 0 || lx >= kTX || ly < 0 || ly >= kTY || x >= S.W || y >= S.H) continue;
      if (!((occ[halo_of(lx >> 1, ly >> 1, lz >> 1)] >> cell_bit(lx, ly, lz)) & 1u)) continue;
      const int64_t g = z * WH + (int64_t)y * S.W + x;
      for (int o = 0; o < 13; o++) {
        int dz, dy, dx;
        back_offset(o, dz, dy, dx);
        if (x + dx >= 0 && x + dx < S.W && y + dy >= 0 && y + dy < S.H) continue;   // a plain step
        const int64_t gn = g + dz * WH + dy * (int64_t)S.W + dx;
        if (gn >= 1 && gn < N && m[gn]) emit(g, gn);
      }
    }
  }
  __syncthreads();
  // 5. staged edges to their global slots
  if (t == 0) {
    const uint32_t ne = min(n_local_edges, (uint32_t)kEdgeBuf);
    edge_base = ne ? atomicAdd(&edge_count[blockIdx.y], (unsigned long long)ne) : 0ull;
  }
  __syncthreads();
  {
    const uint32_t ne = min(n_local_edges, (uint32_t)kEdgeBuf);
    for (uint32_t i = t; i < ne; i += kCclThreads) {
      const unsigned long long j = edge_base + i;
      if ((int64_t)j < S.edge_cap) edges[S.edge + j] = ebuf[i];
    }
  }
  // 6. labels: the component's minimum voxel as a global index, background -> 0.  First
  //    every occupied cell's label, once per cell, into par (whose roots are no longer
  //    needed), then whole rows of voxels from their cells' labels (vector stores).
  for (int cz = 0; cz < ncz; cz++) {
    const int c = (cz * kCY + cy) * kCX + cx;
    if (!occ[halo_of(cx, cy, cz)]) continue;
    const uint32_t r = minv[par[c]];
    par[c] = (uint32_t)((T.z0 + (int)(r / (kTX * kTY))) * WH + (int64_t)(T.y0 + (int)((r / kTX) % kTY)) * S.W +
                        T.x0 + (int)(r % kTX));
  }
  __syncthreads();
  const int lx0 = (t % (kTX / 4)) * 4, ly = t / (kTX / 4);
  const int x = T.x0 + lx0, y = T.y0 + ly;
  if (y >= S.H) return;
  int32_t *L = labels + S.vox;
  const bool vec = x + 3 < S.W && S.W % 4 == 0 && (reinterpret_cast<uintptr_t>(L) & 15u) == 0;
  const int c0x = lx0 >> 1;   // the quad's voxels lie in cells c0x (first two) and c0x + 1
  for (int lz = 0; lz < T.tz; lz++) {
    const int64_t g = (T.z0 + lz) * WH + (int64_t)y * S.W + x;
    const int b = ((lz & 1) << 2) | ((ly & 1) << 1);   // bit of the even-x voxel in its cell
    const uint32_t o0 = occ[halo_of(c0x, ly >> 1, lz >> 1)] >> b, o1 = occ[halo_of(c0x + 1, ly >> 1, lz >> 1)] >> b;
    const int cb = ((lz >> 1) * kCY + (ly >> 1)) * kCX + c0x;
    const int32_t l0 = (o0 & 3u) ? (int32_t)par[cb] : 0, l1 = (o1 & 3u) ? (int32_t)par[cb + 1] : 0;
    int32_t out[4] = {(o0 & 1u) ? l0 : 0, (o0 & 2u) ? l0 : 0, (o1 & 1u) ? l1 : 0, (o1 & 2u) ? l1 : 0};
    if (vec) {
      *reinterpret_cast<int4 *>(L + g) = make_int4(out[0], out[1], out[2], out[3]);
    } else {
#pragma unroll
      for (int k = 0; k < 4; k++)
        if (x + k < S.W) L[g + k] = out[k];
    }
  }
}

// ------------------------------------------------------------------ pass 2: cross-tile edges
__global__ void k_ccl_edges(const Sub *subs, const int2 *edges, const unsigned long long *edge_count,
                            int32_t *labels, int *status) {
  const Sub S = subs[blockIdx.y];
  const unsigned long long cnt = edge_count[blockIdx.y];
  if (cnt > (unsigned long long)S.edge_cap) return;   // overflowed: k_ccl_cross_direct merges instead
  const int64_t n = (int64_t)S.W * S.H * S.D;
  int32_t *L = labels + S.vox;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)cnt;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int2 ab = edges[S.edge + e];
    uf_union(L, ab.x, ab.y, S.walk_limit > 0 ? S.walk_limit : n, status);
  }
}

// The same cross-tile edges straight from the mask, for a substack whose list overflowed.
template <int TZ>
__global__ void __launch_bounds__(kCclThreads) k_ccl_cross_direct(const Sub *subs, const uint8_t *mask,
                                                                 const unsigned long long *edge_count,
                                                                 int32_t *labels, int *status) {
  const Sub S = subs[blockIdx.y];
  if (edge_count[blockIdx.y] <= (unsigned long long)S.edge_cap) return;
  CclTile T;
  if (!ccl_tile<TZ>(S, blockIdx.x, T)) return;
  const int t = threadIdx.x;
  const int lx0 = (t % (kTX / 4)) * 4, ly = t / (kTX / 4);
  const int x = T.x0 + lx0, y = T.y0 + ly;
  if (y >= S.H) return;
  const int64_t WH = (int64_t)S.W * S.H, n = WH * S.D;
  const uint8_t *m = mask + S.vox;
  int32_t *L = labels + S.vox;
  for (int lz = 0; lz < T.tz; lz++) {
    const int z = T.z0 + lz;
    for (int k = 0; k < 4 && x + k < S.W; k++) {
      const int64_t g = z * WH + (int64_t)y * S.W + x + k;
      if (g == 0 || !m[g]) continue;
      for (int o = 0; o < 13; o++) {
        int dz, dy, dx;
        back_offset(o, dz, dy, dx);
        if (!leaves_tile(S, T, x + k, y, z, lx0 + k, ly, lz, dz, dy, dx)) continue;
        const int64_t gn = g + dz * WH + dy * (int64_t)S.W + dx;
        if (gn >= 1 && m[gn]) uf_union(L, (int32_t)g, (int32_t)gn, S.walk_limit > 0 ? S.walk_limit : n, status);
      }
    }
  }
}

// ------------------------------------------------------------------ pass 3: flatten
// 4096 voxels per block, 16 consecutive voxels per thread.  Root bits of voxels
// [32w, 32w+32) of block b go to word (S.blk + b) * 128 + w.
template <bool FROM_LABELS>
__global__ void __launch_bounds__(256) k_ccl_flatten(const Sub *subs, uint8_t *mask, int32_t *labels,
                                                    uint32_t *root_bits, uint32_t *blk_counts, int *status) {
  __shared__ uint32_t wcnt[8];
  const Sub S = subs[blockIdx.y];
  const int64_t n = (int64_t)S.W * S.H * S.D;
  const int64_t base = (int64_t)blockIdx.x * kScanBlock;
  if (base >= n) return;
  const int64_t i0 = base + threadIdx.x * 16;
  int32_t *L = labels + S.vox;
  uint8_t *m = mask + S.vox;
  uint32_t bits = 0;
  if (!FROM_LABELS) {
    uint8_t mk[16];
    if (i0 + 16 <= n && ((reinterpret_cast<uintptr_t>(m + i0) & 15) == 0)) {
      *reinterpret_cast<uint4 *>(mk) = __ldg(reinterpret_cast<const uint4 *>(m + i0));
    } else {
      for (int k = 0; k < 16; k++) mk[k] = (i0 + k < n) ? m[i0 + k] : 0;
    }
    // level by level over the 16 voxels: their labels, then the labels' parents, so the
    // loads of a level are in flight together; deeper walks (labels merged across tiles
    // more than once) continue one by one
    int32_t l[16], p[16];
#pragma unroll
    for (int k = 0; k < 16; k++) l[k] = (mk[k] && i0 + k != 0) ? __ldcg(L + i0 + k) : -1;
#pragma unroll
    for (int k = 0; k < 16; k++) p[k] = l[k] >= 0 ? __ldcg(L + l[k]) : -1;
#pragma unroll
    for (int k = 0; k < 16; k++) {
      if (l[k] < 0) continue;
      const int32_t r = p[k] == l[k] ? l[k] : uf_root(L, p[k], S.walk_limit > 0 ? S.walk_limit : n, status);
      if (r != l[k]) L[i0 + k] = r;
      if (r == (int32_t)(i0 + k)) bits |= 1u << k;
    }
  } else {
    // labels produced elsewhere: foreground = nonzero label, roots label themselves
    for (int k = 0; k < 16; k++) {
      const int64_t i = i0 + k;
      if (i >= n) break;
      const int32_t l = L[i];
      m[i] = l != 0;
      if (i > 0 && l == (int32_t)i) bits |= 1u << k;
    }
  }
  const uint32_t hi = __shfl_down_sync(0xFFFFFFFFu, bits, 1);
  if ((threadIdx.x & 1) == 0) root_bits[(S.blk + blockIdx.x) * (kScanBlock / 32) + threadIdx.x / 2] = bits | (hi << 16);
  uint32_t c = __popc(bits);
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xFFFFFFFFu, c, o);
  if ((threadIdx.x & 31) == 0) wcnt[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
    for (int k = 0; k < 8; k++) tot += wcnt[k];
    blk_counts[S.blk + blockIdx.x] = tot;
  }
}

// The same pass over the fused sweep's foreground list instead of the whole volume (the list
// holds every foreground voxel but voxel 0): root bits and block counts start at zero and
// each root sets its own bit and counts itself.  fg_root holds each entry's voxel index
// (written by the sweep beside the 32-byte entry, so that this pass reads 4 bytes per
// entry) and is overwritten with the entry's root.  A substack whose list overflowed is
// skipped; its batch is redone with the separate passes.
constexpr int kFlatFgPerThread = 16;

__global__ void __launch_bounds__(256) k_ccl_flatten_fg(const Sub *subs, const unsigned long long *fg_count,
                                                       int32_t *labels,
                                                       uint32_t *root_bits, uint32_t *blk_counts, int32_t *fg_root,
                                                       int *status) {
  const Sub S = subs[blockIdx.y];
  const int64_t cnt = (int64_t)fg_count[blockIdx.y * kFgCountStride];
  if (cnt > S.fg_cap) return;
  const int64_t n = (int64_t)S.W * S.H * S.D;
  int32_t *L = labels + S.vox;
  // a warp takes 32 * kFlatFgPerThread consecutive entries, lane l every 32nd from l, so each
  // load and store of the warp covers 32 consecutive entries
  const int lane = threadIdx.x & 31;
  const int64_t span = 32 * kFlatFgPerThread;
  const int64_t stride = ((int64_t)gridDim.x * blockDim.x >> 5) * span;
  for (int64_t w0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * span; w0 < cnt; w0 += stride) {
    const int64_t e0 = w0 + lane;   // entries e0 + 32 k
    // level by level: the entries' voxels, their labels, the labels' parents
    int32_t idx[kFlatFgPerThread], l[kFlatFgPerThread], p[kFlatFgPerThread];
#pragma unroll
    for (int k = 0; k < kFlatFgPerThread; k++) idx[k] = e0 + 32 * k < cnt ? fg_root[S.fg + e0 + 32 * k] : -1;
#pragma unroll
    for (int k = 0; k < kFlatFgPerThread; k++) l[k] = idx[k] >= 0 ? __ldcg(L + idx[k]) : -1;
#pragma unroll
    for (int k = 0; k < kFlatFgPerThread; k++) p[k] = l[k] >= 0 ? __ldcg(L + l[k]) : -1;
#pragma unroll
    for (int k = 0; k < kFlatFgPerThread; k++) {
      if (l[k] < 0) continue;
      const int32_t r = p[k] == l[k] ? l[k] : uf_root(L, p[k], S.walk_limit > 0 ? S.walk_limit : n, status);
      if (r != l[k]) L[idx[k]] = r;
      fg_root[S.fg + e0 + 32 * k] = r;   // the entry's root, read by the region accumulation
      if (r == idx[k]) {
        const int64_t b = idx[k] / kScanBlock;
        const int o = (int)(idx[k] % kScanBlock);
        atomicOr(root_bits + (S.blk + b) * (kScanBlock / 32) + o / 32, 1u << (o % 32));
        atomicAdd(blk_counts + S.blk + b, 1u);
      }
    }
  }
}

// ------------------------------------------------------------------ launchers
void launch_ccl(const Sub *d_subs, int nsub, int max_w, int max_h, int max_d, int64_t max_n, const uint8_t *mask,
                int32_t *labels, int2 *edges, unsigned long long *edge_count, uint32_t *root_bits,
                uint32_t *blk_counts, int *d_status, int num_sms, cudaStream_t s, const FgEntry *fg,
                const unsigned long long *fg_count, int64_t max_fg, int32_t *fg_root) {
  const int64_t cols = (int64_t)ceil_div(max_w, kTX) * ceil_div(max_h, kTY);
  const auto tiles_of = [&](int tz) { return cols * ceil_div(max_d, tz); };
  const int tz = tiles_of(32) * nsub >= 2 * (int64_t)num_sms ? 32 : tiles_of(16) * nsub * 2 >= num_sms ? 16 : 8;
  const dim3 grid((unsigned)tiles_of(tz), nsub);
  auto local = tz == 32 ? k_ccl_local<32> : tz == 16 ? k_ccl_local<16> : k_ccl_local<8>;
  auto cross = tz == 32 ? k_ccl_cross_direct<32> : tz == 16 ? k_ccl_cross_direct<16> : k_ccl_cross_direct<8>;
  KLAUNCH("k_ccl_local", s, (local<<<grid, kCclThreads, 0, s>>>(d_subs, mask, labels, edges, edge_count)));
  const unsigned eb = (unsigned)max(1, (8 * num_sms + nsub - 1) / nsub);
  KLAUNCH("k_ccl_edges", s, (k_ccl_edges<<<dim3(eb, nsub), 256, 0, s>>>(d_subs, edges, edge_count, labels,
                                                                        d_status)));
  KLAUNCH("k_ccl_cross_direct", s, (cross<<<grid, kCclThreads, 0, s>>>(d_subs, mask, edge_count, labels, d_status)));
  if (fg) {
    const int64_t want = std::min((int64_t)ceil_div(max_fg, 256 * kFlatFgPerThread),
                                  (int64_t)(8 * num_sms / (nsub > 0 ? nsub : 1) + 1));
    KLAUNCH("k_ccl_flatten", s, (k_ccl_flatten_fg<<<dim3((unsigned)std::max<int64_t>(want, 1), nsub), 256, 0, s>>>(
                                    d_subs, fg_count, labels, root_bits, blk_counts, fg_root, d_status)));
  } else {
    KLAUNCH("k_ccl_flatten", s, (k_ccl_flatten<false><<<dim3(ceil_div(max_n, kScanBlock), nsub), 256, 0, s>>>(
                                    d_subs, const_cast<uint8_t *>(mask), labels, root_bits, blk_counts, d_status)));
  }
}

void launch_roots_from_labels(const Sub *d_subs, int nsub, int64_t max_n, const int32_t *labels, uint8_t *mask,
                              uint32_t *root_bits, uint32_t *blk_counts, cudaStream_t s) {
  KLAUNCH("k_roots_from_labels", s, (k_ccl_flatten<true><<<dim3(ceil_div(max_n, kScanBlock), nsub), 256, 0, s>>>(
                                        d_subs, mask, const_cast<int32_t *>(labels), root_bits, blk_counts,
                                        nullptr)));
}

}  // namespace hdog
