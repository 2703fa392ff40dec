// Brick allocation: per-pixel projection, row/column de-duplication and the
// parallel octree insert that replaces the reference's sequential traversal
// (transformLoopSimPrecalculatedNeg_subtree, traversal_wrapper_functions.cpp:576-694,
//  queryPointDepthSingle_func_subtree / addLeaf, traversal_functions.cpp:185-211, 308-395).
//
// The reference walks pixels in raster order; three of its outcomes depend on
// that order and are reproduced exactly here:
//   * which pixels are processed (the de-duplication recurrence) -- computed
//     by an exact tiled fixed-point solve of the recurrence;
//   * leaf indices -- assigned in order of the first pixel that created each
//     leaf (sort of pending leaves by first pixel);
//   * parent leaves -- the finest ancestor leaf that existed when the leaf was
//     created, i.e. the finest ancestor with a smaller index.
// Branch indices are assigned in arrival order; they are internal.
#include <cub/cub.cuh>

#include "ff_kernels.h"
#include "ff_sort.h"

namespace ffb {

__device__ __forceinline__ uint32_t ld_volatile(const uint32_t *p) { return *(volatile const uint32_t *)p; }

// Octree read on the descent, cached in L1.  Safe without coherence: a valid
// leaf index or child pointer never changes while the insert runs (they are
// written once; grow() runs between kernels), so a cached read that returns
// one is exact; a slot another thread claims meanwhile may still read as
// BRANCHINIT here, and the atomicCAS that follows returns its current value.
__device__ __forceinline__ uint32_t ld_tree(const uint32_t *p) { return __ldca(p); }

// ---------------------------------------------------------------- bbox ----

// computeBoundingboxIntCPU(ushort), geometryfusion_mipmap_cpu.cpp:1270-1303,
// round-to-nearest float arithmetic in the reference's operation order.
__global__ void k_first_bbox(const uint16_t *depth, int W, int H, CamF p, float scaling, float maxcam, int bw,
                             Counters *cnt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  int mn[3] = {1000000, 1000000, 1000000}, mx[3] = {-1000000, -1000000, -1000000};
  if (i < W * H) {
    int x = i % W, y = i / W;
    float pz = __fmul_rn((float)depth[i], scaling);
    if (pz > 0.0f && pz < maxcam) {
      float px = __fmul_rn(__fdiv_rn(__fsub_rn((float)x, p.cx), p.fx), pz);
      float py = __fmul_rn(__fdiv_rn(__fsub_rn((float)y, p.cy), p.fy), pz);
#pragma unroll
      for (int r = 0; r < 3; r++) {
        float s = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(p.r[3 * r], px), __fmul_rn(p.r[3 * r + 1], py)),
                                      __fmul_rn(p.r[3 * r + 2], pz)),
                            p.t[r]);
        int v = __float2int_rz(s);
        mn[r] = v - bw;
        mx[r] = v + bw;
      }
    }
  }
#pragma unroll
  for (int r = 0; r < 3; r++) {
    int a = mn[r], b = mx[r];
    for (int o = 16; o > 0; o >>= 1) {
      a = min(a, __shfl_xor_sync(0xffffffffu, a, o));
      b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&cnt->box_min[r], a);
      atomicMax(&cnt->box_max[r], b);
    }
  }
}

void launch_first_bbox(const uint16_t *depth, int W, int H, const CamF &p, float scaling, float maxcam, int bw,
                       Counters *cnt, cudaStream_t s) {
  int n = W * H;
  note_launch();
  k_first_bbox<<<(n + 255) / 256, 256, 0, s>>>(depth, W, H, p, scaling, maxcam, bw, cnt);
}

// ------------------------------------------------------------- project ----

// Per pixel: v = (int)(((qx[x] + qy[y]) * depth) * scaling + t), the
// reference's key arithmetic (traversal_wrapper_functions.cpp:613-630,
// addMap's qxp/qyp, geometryfusion_mipmap_cpu.cpp:1807-1822), in
// round-to-nearest with no fused multiply-add.  w = target brick edge in
// voxels, floor(max(depth,1)*8) (leafScaleFunc, inline_functions.hpp:128-145),
// or -1 for invalid depth.
// Voxel coordinates of a pixel's surface point and its target brick scale
// (-1: invalid), under the default rounding: ((qxp+qyp)*d)*scaling + t per
// axis, truncated (traversal_wrapper_functions.cpp:613-630), and
// leafScaleFunc's floor(max(z,1)*8) (inline_functions.hpp:128-145).
__device__ __forceinline__ int4 project_point(float d, float px, float py, const CamF &p, float scaling,
                                              float maxcam) {
  int v[3];
#pragma unroll
  for (int r = 0; r < 3; r++) {
    float qx = __fmul_rn(p.r[3 * r + 0], px);
    float qy = __fadd_rn(__fmul_rn(p.r[3 * r + 1], py), p.r[3 * r + 2]);
    float s = __fadd_rn(__fmul_rn(__fmul_rn(__fadd_rn(qx, qy), d), scaling), p.t[r]);
    v[r] = __float2int_rz(s);
  }
  const float ds = __fmul_rn(d, scaling);
  int target = -1;
  if (ds > 0.0f && ds < maxcam) {
    float f = ds < 1.0f ? 1.0f : ds;
    target = (int)(uint16_t)floorf(__fmul_rn(f, 8.0f));
  }
  return make_int4(v[0], v[1], v[2], target);
}

// ------------------------------------------------------------- dedupe -----
//
// The reference processes pixel (x,y) iff its depth is valid and its brick
// key k = v & -8 differs from s(x,y-1) and from s(x-1,y), where
// s = k if processed and -1 otherwise (traversal_wrapper_functions.cpp:636-639,
// 688-690).  This is a recurrence over the two predecessors only, so it has a
// unique solution.  Each warp solves one tile, 32 pixels wide, exactly, given
// the state of the column to its left and the row above it.  The key
// comparisons never change, so they are made once, as a word per row (bit:
// column): valid V, U = k(x,r)==k(x,r-1), L = k(x,r)==k(x-1,r).  A row is then a
// dozen word operations: a = V & ~(p(r-1) & U), and p(x) = a(x) && !(p(x-1) &&
// L(x)).  p(x) = a(x) where x is not chained to its left neighbour (a & L == 0)
// and alternates along a chain, so p is known from the parity of each chain's
// start, carried along the chain by an addition (solve_row).  Tiles exchange
// their right columns' and bottom rows' p and repeat until none changes; a chain
// of dependencies crosses at most tilesX+tilesY tiles, which bounds the number
// of rounds.

__device__ __forceinline__ void grid_barrier(uint32_t *bar, uint32_t nblocks, Counters *cnt, uint32_t limit) {
  grid_barrier_bounded(bar, nblocks, &cnt->error, ERR_DEDUPE_TIMEOUT, limit);
}

constexpr int DD_WARPS = 8;  // tiles (warps) per block
// Blocks that share one launch, per SM.  A launch's tiles must all be resident, and
// frames that do not fit one launch pay its rounds of barriers again, so as
// many blocks as the registers allow without spilling in the rows' loop: 64 a
// thread, 256 threads, four blocks fill the register file (the launch bounds below
// keep them resident; their scratch is 147 of the 228 KB).  4,736 tiles a launch:
// eight maps of mixed sizes (3,750 tiles of 32 rows) take 74 us; at three blocks,
// in two launches, 91.
constexpr int DD_BLOCKS_PER_SM = 4;
// the largest image, in warps per SM
constexpr int DD_IMAGE_WARPS_PER_SM = 24;
// tile height: 16 rows (more, shorter tiles shorten each warp's chain of
// rows), or 32 when the image has more 16-row tiles than resident warps
constexpr int DD_ROWS_SHORT = 16, DD_ROWS_TALL = 32;
constexpr int DD_ROWS_LOW = 8;  // more, shorter tiles again (a tuning choice)

__device__ __forceinline__ bool same3(int a0, int a1, int a2, int b0, int b1, int b2) {
  return a0 == b0 && a1 == b1 && a2 == b2;
}

// p of a row from a and the chained positions c (c & ~a == 0, bit 0 not in c).
// A chain's p is 1 at every second position from its start, the first one where
// a(start) is 1, the next where it is 0: even positions for starts in q, odd
// ones for the others.  The addition of the lowest chained position above a start
// in q carries through that chain, and clears it.
__device__ __forceinline__ uint32_t solve_row(uint32_t a, uint32_t c) {
  constexpr uint32_t EVEN = 0x55555555u;
  const uint32_t q = ~c & ~(a ^ EVEN);
  const uint32_t e = q | (c & ~(c + ((q << 1) & c)));
  return ~(e ^ EVEN);
}

// The cells the processed pixels ask for.  A descent of the octree ends at the
// cell of edge h that holds the pixel's voxel (h: the smallest power of two
// not below the pixel's target, at most half the volume), and pixels of the
// same cell make the same descent: only the cell's first pixel matters to its
// leaf's index, and half the pixels of a surface are processed, some hundred
// per cell.  So each tile lists its cells, with the first pixel that asked, for
// the insert to look up.  A cell may be listed more than once (its pixels in two
// tiles, or a hash slot taken over): the insert keeps the smallest pixel.
constexpr int CELL_TAB = 64;
template <int DD_ROWS>
struct TileScratch {
  uint16_t depth[DD_ROWS][32];
  uint16_t item[DD_ROWS * 32];       // pixels to look at: 32 row + column
  unsigned long long tab[CELL_TAB];  // cells listed, by hash; a later one of the same slot takes it over
};

// Lane r's word of row r's processed pixels, less those that share a cell with
// an earlier processed pixel two steps away: same-cell steps to the left (SL)
// and up (SU), in the tile.  Processed pixels of a cell are two steps apart (a
// neighbour of the same cell is not processed), so about one per cell is left.
__device__ __forceinline__ uint32_t first_of_cells(uint32_t P, uint32_t SL, uint32_t SU, int lane) {
  const uint32_t full = 0xffffffffu;
  uint32_t P1 = __shfl_up_sync(full, P, 1), SL1 = __shfl_up_sync(full, SL, 1), SU1 = __shfl_up_sync(full, SU, 1);
  uint32_t P2 = __shfl_up_sync(full, P, 2);
  if (lane < 1) P1 = SL1 = SU1 = 0;
  if (lane < 2) P2 = 0;
  const uint32_t ll = SL & (SL << 1) & (P << 2), lu = SL & (SU << 1) & (P1 << 1);
  const uint32_t uu = SU & SU1 & P2, ul = SU & SL1 & (P1 << 1), ur = SU & (SL1 >> 1) & (P1 >> 1);
  return P & ~(ll | lu | uu | ul | ur);
}

// List the cells of a tile's pixels in `word` (lane r: row r), rows top to bottom
// and columns left to right.  True if any of the pixels lies within a brick of
// where the frame's bounding box leaves the volume.
template <int DD_ROWS>
__device__ __forceinline__ bool list_cells(const MapFrame &F, TileScratch<DD_ROWS> &T, int x0, int y0, uint32_t word,
                                           float px, float py_lane) {
  const int lane = threadIdx.x & 31;
  const uint32_t full = 0xffffffffu;
  uint32_t at = (uint32_t)__popc(word);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(full, at, o);
    if (lane >= o) at += t;
  }
  const uint32_t total = __shfl_sync(full, at, 31);
  at -= (uint32_t)__popc(word);
  for (uint32_t w = word; w; w &= w - 1) T.item[at++] = (uint16_t)(32 * lane + __ffs(w) - 1);
  for (int k = lane; k < CELL_TAB; k += 32) T.tab[k] = ~0ull;
  __syncwarp();
  const CamF cam = F.p;
  const float scaling = F.scaling, maxcam = F.maxcam;
  const uint32_t n = F.n;
  const bool pow2 = (n & (n - 1)) == 0;
  const int margin = (int)F.bw + 7;
  bool near_face = false;
  uint32_t kept = 0;
  // (two or four groups of pixels at a time were slower: the code runs once or
  // twice a launch, and what it waits for is its own instructions)
  for (uint32_t j0 = 0; j0 < total; j0 += 32) {
    const bool have = j0 + lane < total;
    const int code = have ? T.item[j0 + lane] : 0;
    const int r = code >> 5, c = code & 31;
    const float ix = __shfl_sync(full, px, c), iy = __shfl_sync(full, py_lane, r);
    const int4 v = project_point((float)T.depth[r][c], ix, iy, cam, scaling, maxcam);
    near_face |= have && (min(v.x, min(v.y, v.z)) < margin || max(v.x, max(v.y, v.z)) >= (int)n - margin);
    const uint32_t cx = (uint16_t)v.x, cy = (uint16_t)v.y, cz = (uint16_t)v.z, target = (uint32_t)v.w;
    bool add = have && v.x >= 0 && cx < n && v.y >= 0 && cy < n && v.z >= 0 && cz < n;
    // (a volume whose side is no power of two has no such cells: voxel and target name the descent)
    uint32_t lg = target;
    int sh = 0;
    if (pow2) {
      lg = min(32 - __clz(target - 1), 30 - __clz(n));
      sh = (int)lg & 31;
    }
    const uint32_t k0 = (cx >> sh) | (cy >> sh) << 16, k1 = (cz >> sh) | lg << 16;
    const unsigned long long key = (unsigned long long)k1 << 32 | k0;
    const uint32_t slot = ((k0 ^ k1 * 0x85EBCA6Bu) * 0x9E3779B1u) >> 26;
    add = add && T.tab[slot] != key;
    // the first pixel of each key not listed yet (few: a shuffle each)
    unsigned f = 0;
    for (unsigned m = __ballot_sync(full, add); m;) {
      const int lead = __ffs(m) - 1;
      const unsigned long long lead_key = __shfl_sync(full, key, lead);
      m &= ~__ballot_sync(full, key == lead_key);
      f |= 1u << lead;
    }
    if (!f) continue;
    if ((f >> lane) & 1u) {
      T.tab[slot] = key;
      T.item[kept + __popc(f & ((1u << lane) - 1u))] = (uint16_t)code;  // (at or before this pass's items)
    }
    kept += (uint32_t)__popc(f);
    __syncwarp();
  }
  near_face = __any_sync(full, near_face);
  if (!kept) return near_face;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&F.cnt->cands, kept);
  base = __shfl_sync(full, base, 0);
  for (uint32_t j0 = 0; j0 < kept; j0 += 32) {
    const int code = j0 + lane < kept ? T.item[j0 + lane] : 0;
    const int r = code >> 5, c = code & 31;
    const float ix = __shfl_sync(full, px, c), iy = __shfl_sync(full, py_lane, r);
    const int4 v = project_point((float)T.depth[r][c], ix, iy, cam, scaling, maxcam);
    if (j0 + lane < kept)
      F.cand[base + j0 + lane] =
          make_uint4((uint32_t)(uint16_t)v.x | (uint32_t)(uint16_t)v.y << 16,
                     (uint32_t)(uint16_t)v.z | (uint32_t)v.w << 16, (uint32_t)(y0 + r) * (uint32_t)F.W + (uint32_t)(x0 + c), 0u);
  }
  return near_face;
}

// Same-cell words of a tile whose pixels have several cell sizes: lane r's row's
// U and L, less the steps between pixels of different sizes.
template <int DD_ROWS>
__device__ __forceinline__ void same_size(const TileScratch<DD_ROWS> &T, float scaling, float maxcam, uint32_t &SU,
                                          uint32_t &SL) {
  const int lane = threadIdx.x & 31;
  int above = -1;
#pragma unroll 2
  for (int r = 0; r < DD_ROWS; r++) {
    const int4 v = project_point((float)T.depth[r][lane], 0.0f, 0.0f, CamF(), scaling, maxcam);
    const int lg = v.w < 0 ? -1 : __clz(v.w - 1);
    const int left = __shfl_up_sync(0xffffffffu, lg, 1);
    const uint32_t eu = __ballot_sync(0xffffffffu, lg == above), el = __ballot_sync(0xffffffffu, lg == left);
    if (lane == r) SU &= eu, SL &= el;
    above = lg;
  }
}

// A tile whose pixels come close to the volume's faces: the frame's bounding
// box over its processed pixels (lane r's word: row r).
template <int DD_ROWS>
__device__ __forceinline__ void tile_box(const MapFrame &F, const TileScratch<DD_ROWS> &T, int rows, uint32_t word,
                                         float px, float py_lane) {
  const int lane = threadIdx.x & 31;
  const int n = (int)F.n, bw = (int)F.bw;
  int lo[3] = {0, 0, 0}, hi[3] = {n - 1, n - 1, n - 1};
#pragma unroll 1
  for (int r = 0; r < rows; r++) {
    const uint32_t row = __shfl_sync(0xffffffffu, word, r);
    const float py = __shfl_sync(0xffffffffu, py_lane, r);
    if (!((row >> lane) & 1u)) continue;
    const int4 v = project_point((float)T.depth[r][lane], px, py, F.p, F.scaling, F.maxcam);
    const int vv[3] = {v.x, v.y, v.z};
#pragma unroll
    for (int a = 0; a < 3; a++) lo[a] = min(lo[a], vv[a] - bw), hi[a] = max(hi[a], vv[a] + bw);
  }
  __syncwarp();
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int l = __reduce_min_sync(0xffffffffu, lo[a]), h = __reduce_max_sync(0xffffffffu, hi[a]);
    if (lane == 0 && l < 0) atomicMin(&F.cnt->box_min[a], l);
    if (lane == 0 && h >= n) atomicMax(&F.cnt->box_max[a], h);
  }
}

// Tiles are 32 pixels wide and DD_ROWS high, a warp each.  bnd: processed bits
// of the right column and of the bottom row, [2 rounds][ntiles] each.
// bar: [0] arrivals, [1] generation, [4..6] per-round change counters (rotating)
// One launch for all frames of a batch: warps are dealt out over the maps'
// tiles in order; the rounds and their barrier are shared (a map whose tiles
// have settled recomputes the same bits until every map has).
// Maps [m0, m1) of the batch (their tiles must all be resident at once).
//
// What bounds it: latency -- a few warps per scheduler, three to five rounds
// with a grid barrier (2 us) each.  A row of a tile used to be solved across the
// lanes with two ballots and a search for the chain's start (240 ns a row); the
// word operations take 20 ns and leave the barriers.  With the list of cells
// (5 us) a 640x480 frame's launch takes 24 us (37 before, without a list), ten
// frames' 51 us (64), ten 1280x960 frames' launches 244 us (336).
template <int DD_ROWS>
__device__ __forceinline__ void dedupe_body(const BatchDesc *__restrict__ bd, const TileEnds &ends, int m0, int m1,
                                            uint32_t *bar) {
  __shared__ TileScratch<DD_ROWS> scratch[DD_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t base = m0 ? ends.end[m0 - 1] : 0u;
  const uint32_t gtile = base + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  int m = m0;
  while (m < m1 - 1 && gtile >= ends.end[m]) m++;
  const bool active = gtile < ends.end[m1 - 1];  // (the others only join the barriers)
  const MapFrame &F = bd->f[m];
  const int tile = (int)(gtile - (m ? ends.end[m - 1] : 0u));
  const uint16_t *__restrict__ depth = F.depth;
  const CamF cam = F.p;
  const float scaling = F.scaling, maxcam = F.maxcam;
  const int W = F.W, H = F.H, tilesX = F.tilesX, tilesY = F.tilesY;
  const int ntiles = tilesX * tilesY;
  uint32_t *pR = F.bnd, *pB = pR + 2 * (size_t)ntiles;
  const int tx = active ? tile % tilesX : 0, ty = active ? tile / tilesX : 0;
  const int x0 = tx * 32, y0 = ty * DD_ROWS, x = x0 + lane;
  // each map's counters for this frame (read from the first barrier on)
  if (blockIdx.x == 0 && (int)threadIdx.x < m1 - m0) {
    const MapFrame &G = bd->f[m0 + threadIdx.x];
    Counters *c = G.cnt;
    // (not the confidence network's error word, which that network may be
    // setting meanwhile on another stream)
    constexpr int keep = (int)(offsetof(Counters, cnn_error) / 4);
    uint32_t *w = reinterpret_cast<uint32_t *>(c);
    for (int k = 0; k < (int)(sizeof(Counters) / 4); k++)
      if (k != keep) w[k] = 0;
    c->branches_used = G.branches_init;
    for (int r = 0; r < 3; r++) {
      c->box_min[r] = 0;
      c->box_max[r] = (int)G.n - 1;
    }
  }
  const int rows = active ? min(DD_ROWS, H - y0) : 0;
  // Project the tile and make the key comparisons: the tile's depth and the row
  // above it, and (a lane per row) the column to its left.
  const bool col_ok = active && x < W;
  const bool row_ok = lane < rows, left_ok = row_ok && tx > 0;
  const uint16_t *dcol = depth + (size_t)y0 * W + x;
  TileScratch<DD_ROWS> &T = scratch[warp];
  uint16_t d_above = 0, d_left = 0;
  if (col_ok && ty > 0) d_above = __ldg(dcol - W);
  if (left_ok) d_left = __ldg(&depth[(size_t)(y0 + lane) * W + x0 - 1]);
  uint16_t dv[DD_ROWS];
#pragma unroll
  for (int r = 0; r < DD_ROWS; r++) dv[r] = col_ok && r < rows ? __ldg(dcol + (size_t)r * W) : (uint16_t)0;
  const float px = col_ok ? __ldg(&F.pxp[x]) : 0.0f;
  const float px_left = left_ok ? __ldg(&F.pxp[x0 - 1]) : 0.0f;
  const float py_lane = row_ok ? __ldg(&F.pyp[y0 + lane]) : 0.0f;
  const float py_above = active && ty > 0 ? __ldg(&F.pyp[y0 - 1]) : 0.0f;
#pragma unroll
  for (int r = 0; r < DD_ROWS; r++) T.depth[r][lane] = dv[r];
  __syncwarp();
  const float px_first = __shfl_sync(0xffffffffu, px, 0);
  // this lane's row: its first pixel has the key of the left tile's last one
  bool eq_left = false;
  if (left_ok) {
    const int4 a = project_point((float)d_left, px_left, py_lane, cam, scaling, maxcam);
    const int4 b = project_point((float)T.depth[lane][0], px_first, py_lane, cam, scaling, maxcam);
    eq_left = same3(a.x & -8, a.y & -8, a.z & -8, b.x & -8, b.y & -8, b.z & -8);
  }
  uint32_t V = 0, U = 0, L = 0;  // the masks of row `lane`
  int4 u = project_point((float)d_above, px, py_above, cam, scaling, maxcam);  // the row before
  uint32_t target_min = 0xffffffffu;  // (an invalid pixel's is -1)
  int target_max = -1;
#pragma unroll 4
  for (int r = 0; r < DD_ROWS; r++) {
    const float py = __shfl_sync(0xffffffffu, py_lane, r);
    const int4 v = project_point((float)T.depth[r][lane], px, py, cam, scaling, maxcam);  // (invalid past the image: depth 0)
    const int l0 = __shfl_up_sync(0xffffffffu, v.x, 1);
    const int l1 = __shfl_up_sync(0xffffffffu, v.y, 1);
    const int l2 = __shfl_up_sync(0xffffffffu, v.z, 1);
    const int du = (v.x ^ u.x) | (v.y ^ u.y) | (v.z ^ u.z), dl = (v.x ^ l0) | (v.y ^ l1) | (v.z ^ l2);
    const uint32_t rv = __ballot_sync(0xffffffffu, v.w >= 0);
    const uint32_t ru = __ballot_sync(0xffffffffu, (du & -8) == 0);
    const uint32_t rl = __ballot_sync(0xffffffffu, (dl & -8) == 0) & ~1u;
    if (lane == r) V = rv, U = ru, L = rl;
    target_min = min(target_min, (uint32_t)v.w);
    target_max = max(target_max, v.w);
    u = v;
  }
  // the tile's pixels ask for cells of one size
  const bool one_size = __clz((int)__reduce_min_sync(0xffffffffu, target_min) - 1) ==
                        __clz(__reduce_max_sync(0xffffffffu, target_max) - 1);
  uint32_t word = 0;  // the processed pixels of row `lane`
  uint32_t last_r = 0, last_b = 0, last_left = 0, last_above = 0;
  const int max_rounds = bd->max_rounds;
  volatile uint32_t *chg = bar + 4;
  int round = 0;
  bool converged = false;
  for (; round < max_rounds; round++) {
    const int in = round & 1, out = in ^ 1;
    int changed = 0;
    if (active) {
      uint32_t left_p = 0, above_p = 0;
      if (round > 0) {
        if (tx > 0) left_p = __ldcg(&pR[(size_t)in * ntiles + tile - 1]);
        if (ty > 0) above_p = __ldcg(&pB[(size_t)in * ntiles + tile - tilesX]);
      }
      if (round == 0 || left_p != last_left || above_p != last_above) {
        const uint32_t vl = V & ~((left_p >> lane) & (uint32_t)eq_left);  // (chained to a processed pixel of the left tile)
        uint32_t p = above_p, rb = 0, bb = 0;
#pragma unroll 8
        for (int r = 0; r < DD_ROWS; r++) {
          const uint32_t rv = __shfl_sync(0xffffffffu, vl, r), ru = __shfl_sync(0xffffffffu, U, r),
                         rl = __shfl_sync(0xffffffffu, L, r);
          const uint32_t a = rv & ~(p & ru);
          p = solve_row(a, a & rl);
          rb |= (p >> 31) << r;
          if (r == rows - 1) bb = p;
          if (lane == r) word = p;
        }
        changed = round == 0 || rb != last_r || bb != last_b;
        last_r = rb;
        last_b = bb;
        last_left = left_p;
        last_above = above_p;
      }
      if (lane == 0) {
        pR[(size_t)out * ntiles + tile] = last_r;
        pB[(size_t)out * ntiles + tile] = last_b;
      }
    }
    if (changed && lane == 0) atomicAdd((uint32_t *)&chg[round % 3], 1u);
    // counter (round + 1) % 3 was last read before the previous barrier
    if (blockIdx.x == 0 && threadIdx.x == 0) chg[(round + 1) % 3] = 0;
    // a barrier that gives up marks the first map; every map's frame reports it
    grid_barrier(bar, gridDim.x, bd->f[m0].cnt, bd->f[m0].spin_limit);
    const uint32_t any = chg[round % 3];
    if (!any) {
      converged = true;
      break;
    }
    if (*(volatile uint32_t *)&bd->f[m0].cnt->error & ERR_DEDUPE_TIMEOUT) break;
  }
  // leave the barrier words as the next launch needs them: the arrival count
  // is zero after every completed barrier, counter (round + 1) % 3 was zeroed
  // in this round and counter round % 3 read as zero, and counter
  // (round + 2) % 3 was last read before this round's barrier (after a
  // barrier that gave up or no convergence, the host clears the words)
  if (converged && blockIdx.x == 0 && threadIdx.x == 0) chg[(round + 2) % 3] = 0;
  // the frame's processed pixels, counted once per tile
  const uint32_t nproc = __reduce_add_sync(0xffffffffu, active ? (uint32_t)__popc(word) : 0u);
  if (active && lane == 0 && nproc) atomicAdd(&F.cnt->processed, nproc);
  if (active && converged && nproc) {
    uint32_t look = word;
    if ((F.n & (F.n - 1)) == 0) {  // (else there are no cells, see list_cells)
      uint32_t SU = U, SL = L;
      if (!one_size) same_size(T, scaling, maxcam, SU, SL);
      look = first_of_cells(word, SL, SU, lane);
    }
    const bool near_face = list_cells(F, T, x0, y0, look, px, py_lane);
    if (near_face) tile_box(F, T, rows, word, px, py_lane);
  }
  if (blockIdx.x == 0 && (int)threadIdx.x < m1 - m0) {
    Counters *c = bd->f[m0 + threadIdx.x].cnt;
    c->dedupe_iters = round + 1;
    if (!converged) atomicOr(&c->error, ERR_DEDUPE_NOT_CONVERGED);
    if (*(volatile uint32_t *)&bd->f[m0].cnt->error & ERR_DEDUPE_TIMEOUT) atomicOr(&c->error, ERR_DEDUPE_TIMEOUT);
  }
}

template <int DD_ROWS>
// (a 10-frame sequence of 640x480 frames fits one cooperative launch)
__global__ void __launch_bounds__(32 * DD_WARPS, DD_BLOCKS_PER_SM) k_dedupe(
    const BatchDesc *__restrict__ bd, const __grid_constant__ TileEnds ends, int m0, int m1, uint32_t *bar) {
  dedupe_body<DD_ROWS>(bd, ends, m0, m1, bar);
}

// One map's frame, its descriptor a launch parameter: block 0 also stores it
// to `out`, where the frame's later kernels read it.
template <int DD_ROWS>
__global__ void __launch_bounds__(32 * DD_WARPS, DD_BLOCKS_PER_SM) k_dedupe_one(const __grid_constant__ BatchDesc1 desc,
                                                              BatchDesc *out, uint32_t *bar) {
  if (blockIdx.x == 0) {
    const uint2 *src = reinterpret_cast<const uint2 *>(&desc);
    uint2 *dst = reinterpret_cast<uint2 *>(out);
    for (int k = threadIdx.x; k < (int)(sizeof(BatchDesc1) / 8); k += blockDim.x) dst[k] = src[k];
  }
  dedupe_body<DD_ROWS>(reinterpret_cast<const BatchDesc *>(&desc), desc.ends, 0, 1, bar);
}

int dedupe_tiles(int W, int H, int *tilesX, int *tilesY, int rows) {
  const int tx = (W + 31) / 32, ty = (H + rows - 1) / rows;
  if (tilesX) *tilesX = tx;
  if (tilesY) *tilesY = ty;
  return tx * ty;
}

size_t dedupe_boundary_elems(int W, int H) {
  // sized for the lowest tiles (the largest count)
  return 4 * (size_t)dedupe_tiles(W, H, nullptr, nullptr, DD_ROWS_LOW);
}

// Tiles that one launch takes: the warps that the launch bounds keep resident.
cudaError_t dedupe_capacity(int device, uint32_t &tiles, uint32_t *image_tiles) {
  int sms = 0;
  const cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  tiles = (uint32_t)(sms * DD_BLOCKS_PER_SM * DD_WARPS);
  if (image_tiles) *image_tiles = (uint32_t)(sms * DD_IMAGE_WARPS_PER_SM);
  return e;
}

cudaError_t launch_dedupe(const BatchDesc *h_batch, const BatchDesc *d_batch, int m0, int m1, uint32_t tiles, int rows, uint32_t *barrier,
                          int device, cudaStream_t s) {
  uint32_t cap = 0;
  cudaError_t e = dedupe_capacity(device, cap);
  if (e != cudaSuccess) return e;
  // one warp per tile, all resident at once
  const int blocks = (int)((tiles + DD_WARPS - 1) / DD_WARPS);
  if ((uint32_t)blocks * DD_WARPS > cap || blocks < 1) return cudaErrorInvalidConfiguration;
  TileEnds ends = h_batch->ends;
  void *args[] = {(void *)&d_batch, (void *)&ends, (void *)&m0, (void *)&m1, (void *)&barrier};
  note_launch();
  const void *fn = rows == DD_ROWS_SHORT  ? (const void *)k_dedupe<DD_ROWS_SHORT>
                   : rows == DD_ROWS_LOW ? (const void *)k_dedupe<DD_ROWS_LOW>
                                         : (const void *)k_dedupe<DD_ROWS_TALL>;
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(32 * DD_WARPS), args, 0, s);
}

cudaError_t launch_dedupe_one(const BatchDesc *h_desc, BatchDesc *d_batch, uint32_t tiles, int rows,
                              uint32_t *barrier, int device, cudaStream_t s) {
  uint32_t cap = 0;
  cudaError_t e = dedupe_capacity(device, cap);
  if (e != cudaSuccess) return e;
  const int blocks = (int)((tiles + DD_WARPS - 1) / DD_WARPS);
  if ((uint32_t)blocks * DD_WARPS > cap || blocks < 1 || h_desc->n != 1) return cudaErrorInvalidConfiguration;
  BatchDesc1 d1;
  memcpy(&d1, h_desc, sizeof(BatchDesc1));
  void *args[] = {(void *)&d1, (void *)&d_batch, (void *)&barrier};
  note_launch();
  const void *fn = rows == DD_ROWS_SHORT  ? (const void *)k_dedupe_one<DD_ROWS_SHORT>
                   : rows == DD_ROWS_LOW ? (const void *)k_dedupe_one<DD_ROWS_LOW>
                                         : (const void *)k_dedupe_one<DD_ROWS_TALL>;
  return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(32 * DD_WARPS), args, 0, s);
}

// -------------------------------------------------------------- insert ----

__device__ __forceinline__ void queue_leaf(uint32_t leaf, uint32_t frame, uint32_t *stamp, uint32_t *queue,
                                           Counters *cnt) {
  // coarse leaves lie on the paths of many pixels: a plain read first keeps
  // those repeats off the atomic unit (the exchange below decides the winner)
  if (ld_volatile(&stamp[leaf]) == frame) return;
  if (atomicExch(&stamp[leaf], frame) != frame) {
    uint32_t q = atomicAdd(&cnt->queued, 1u);
    queue[q] = leaf;
  }
}

// The second half of queue_leaf for a leaf whose stamp was read earlier (st):
// the insert's descent reads a level's stamp, then issues the next level's
// octree loads before it looks at the value, so that the two round trips
// overlap.
__device__ __forceinline__ void queue_leaf_after(uint32_t leaf, uint32_t st, uint32_t frame, uint32_t *stamp,
                                                 uint32_t *queue, Counters *cnt) {
  if (st == frame) return;
  if (atomicExch(&stamp[leaf], frame) != frame) {
    uint32_t q = atomicAdd(&cnt->queued, 1u);
    queue[q] = leaf;
  }
}

// Wait until another thread finished allocating tree[ptr]; bounded.
__device__ __forceinline__ uint32_t wait_unlocked(uint32_t *tree, uint32_t ptr, uint32_t cur, Counters *cnt,
                                                  bool *ok, uint32_t limit) {
  uint32_t spins = 0;
  while (cur == LOCKED) {
    if (spins++ >= limit) {
      atomicOr(&cnt->error, ERR_SPIN_TIMEOUT);
      *ok = false;
      return cur;
    }
    __nanosleep(20);
    cur = ld_volatile(tree + ptr);
  }
  return cur;
}

// Branches on one descent's path: at most one per halving of the volume's
// side (16 bits of voxel coordinates) plus the root.
constexpr int DESCENT_MAX = 18;

// One cell of the frame F's list (a voxel v in it, the target, its first pixel
// i): the descent of queryPointDepthSingle_func_subtree: queue the existing
// coarser leaves on the path, allocate missing branches, claim the final leaf.
// Returns the number of octree levels probed; sets *created when it wrote a
// new branch or leaf slot into the octree, and records the branches it passed
// (root first) in path[0, *npath).
__device__ __forceinline__ uint32_t insert_descend(const MapFrame &F, uint32_t i, uint32_t x, uint32_t y, uint32_t z,
                                                   uint32_t target, Counters *cnt, bool *created, uint32_t *path,
                                                   int *npath) {
  const uint32_t n = F.n;
  uint32_t *tree = F.tree;
  const uint32_t leaves_max = F.leaves_max, branches_max = F.branches_max, frame = F.frame;
  uint32_t *stamp = F.stamp, *queue = F.queue;
  PendingLeaf *pend = F.pend;
  const uint32_t pend_cap = F.pend_cap;
  uint32_t probed = 0;
  uint32_t ox = 0, oy = 0, oz = 0;
  uint32_t half = (uint16_t)(n >> 1);
  uint32_t branch = 0;
  bool ok = true;
  // the previous level's leaf (if any) and its stamp, read but not yet looked at
  uint32_t prev_leaf = BRANCHINIT, prev_st = frame;
  int np = 0;
  while ((half >> 1) >= target) {
    probed++;
    if (np < DESCENT_MAX) path[np++] = branch;
    *npath = np;
    uint32_t co = (x >= ox + half) * 1u + (y >= oy + half) * 2u + (z >= oz + half) * 4u;
    uint32_t ptr = branch + co + 8;
    uint32_t leaf = ld_tree(tree + ptr - 8);
    uint32_t child = ld_tree(tree + ptr);
    if (prev_leaf < leaves_max) queue_leaf_after(prev_leaf, prev_st, frame, stamp, queue, cnt);
    prev_leaf = leaf;
    prev_st = leaf < leaves_max ? ld_volatile(&stamp[leaf]) : frame;
    if (child == BRANCHINIT) {
      uint32_t old = atomicCAS(tree + ptr, BRANCHINIT, LOCKED);
      if (old == BRANCHINIT) {
        uint32_t nb = atomicAdd(&cnt->branches_used, 16u);
        if (nb + 16 > branches_max) {
          atomicOr(&cnt->error, ERR_BRANCH_OVERFLOW);
          atomicExch(tree + ptr, BRANCHINIT);
          if (prev_leaf < leaves_max) queue_leaf_after(prev_leaf, prev_st, frame, stamp, queue, cnt);
          return probed;
        }
        // (no fence: a new branch's slots hold BRANCHINIT since an earlier
        // launch, and nothing else this thread wrote is read through it)
        atomicExch(tree + ptr, nb);
        child = nb;
        *created = true;
        if (probed <= (uint32_t)MESH_TOP_LEVELS) atomicOr(&cnt->top_created, 1u);
      } else {
        child = old;
      }
    }
    child = wait_unlocked(tree, ptr, child, cnt, &ok, F.spin_limit);
    if (!ok || child == BRANCHINIT) {
      if (prev_leaf < leaves_max) queue_leaf_after(prev_leaf, prev_st, frame, stamp, queue, cnt);
      return probed;
    }
    ox += half * ((co & 1) != 0);
    oy += half * ((co & 2) != 0);
    oz += half * ((co & 4) != 0);
    branch = child;
    half >>= 1;
  }
  uint32_t co = (x >= ox + half) * 1u + (y >= oy + half) * 2u + (z >= oz + half) * 4u;
  uint32_t ptr = branch + co;
  probed++;
  if (np < DESCENT_MAX) path[np++] = branch;
  *npath = np;
  uint32_t cur = ld_tree(tree + ptr);
  if (prev_leaf < leaves_max) queue_leaf_after(prev_leaf, prev_st, frame, stamp, queue, cnt);
  if (cur == BRANCHINIT) {
    uint32_t old = atomicCAS(tree + ptr, BRANCHINIT, LOCKED);
    if (old == BRANCHINIT) {
      uint32_t rec = atomicAdd(&cnt->pending, 1u);
      if (rec >= pend_cap) {
        atomicOr(&cnt->error, ERR_PENDING_OVERFLOW);
        atomicExch(tree + ptr, BRANCHINIT);
        return probed;
      }
      PendingLeaf pl;
      pl.slot = ptr;
      pl.first_pixel = i;
      pl.pos = make_ushort4((uint16_t)(ox + half * ((co & 1) != 0)), (uint16_t)(oy + half * ((co & 2) != 0)),
                            (uint16_t)(oz + half * ((co & 4) != 0)), (uint16_t)(half / BL));
      pend[rec] = pl;
      __threadfence();
      atomicExch(tree + ptr, PENDING + rec);
      *created = true;
      if (probed <= (uint32_t)MESH_TOP_LEVELS) atomicOr(&cnt->top_created, 1u);
      return probed;
    }
    cur = old;
  }
  cur = wait_unlocked(tree, ptr, cur, cnt, &ok, F.spin_limit);
  if (!ok) return probed;
  if (cur >= PENDING && cur < PENDING + pend_cap) {
    atomicMin(&pend[cur - PENDING].first_pixel, i);
  } else if (cur < leaves_max) {
    queue_leaf(cur, frame, stamp, queue, cnt);
  }
  return probed;
}

// Mark every branch on the descent's path (root first, down to the branch
// that holds the cell's slot, or to the last one reached when the descent
// stopped early) with the frame: the branches whose subtree gained a branch
// or a leaf.  Only cells that created something do it; the loads of the
// stamps are independent, so they overlap.
__device__ __forceinline__ void stamp_path(const MapFrame &F, const uint32_t *path, int np) {
  for (int k = 0; k < np; k++) {
    uint32_t *b = F.bstamp + (path[k] >> 4);
    if (*b != F.frame) *b = F.frame;
  }
}

// Deferred update: mark each brick of the frame's queue (nq entries: the
// q0 the insert queued, then the new leaves in rank order, indices from
// leaves_before) with the frame's bit, and list the bricks no earlier frame
// of the pass has marked.  Thread t of `threads` (whole warps; every thread of
// a warp runs the same number of iterations, so the list slots are claimed with
// one atomic per warp).
__device__ __forceinline__ void mark_queue(const MapFrame &F, uint32_t q0, uint32_t nq, uint32_t leaves_before,
                                           uint32_t t, uint32_t threads) {
  const uint32_t bit = 1u << F.upd_slot;
  for (uint32_t j0 = t & ~31u; j0 < nq; j0 += threads) {
    const uint32_t j = j0 + (t & 31u);
    bool add = false;
    uint32_t b = 0;
    if (j < nq) {
      b = j < q0 ? F.queue[j] : leaves_before + (j - q0);
      // a part of a sharded map updates the bricks it owns; the queue holds
      // each brick once, so the old mask lacks this bit
      if (F.shards <= 1 || owns_brick(F, F.leaf[b])) add = atomicOr(&F.upd_mask[b], bit) == 0u;
    }
    const unsigned ball = __ballot_sync(0xffffffffu, add);
    uint32_t at = 0;
    if ((t & 31) == 0 && ball) at = atomicAdd(F.upd_count, (uint32_t)__popc(ball));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (add) F.upd_list[at + __popc(ball & ((1u << (t & 31)) - 1u))] = b;
  }
}

// Blocks of a chained frame's insert that mark the frame before it, whose leaves
// are placed by then: four dependent round trips (4 us) that the chain of
// frames would wait for in that frame's finalisation overlap the descents here.
constexpr int MARK_BLOCKS = 8;

// The cells the frames' de-duplication listed: blocks over x stride over a
// frame's list, y is the frame of the batch.  Bound by the latency of a descent
// (some eight dependent octree reads): a thread per processed pixel, 140,000 of
// a 640x480 frame where the list has 3,000 to 4,000 cells, took 27.6 us with its
// launch and 80.9 us at 1280x960; the list takes 12.4 and 12.7 us.  At most 40 registers: six
// 256-thread blocks per SM instead of five (a few bytes of spill), for any
// block size the tuning picks.
__global__ void __maxnreg__(40) k_insert(const BatchDesc *__restrict__ bd, int m0, int markers) {
  pdl_enter();
  const uint32_t blocks = gridDim.x - (uint32_t)markers;
  if (blockIdx.x >= blocks) {
    const MapFrame &P = bd->f[m0 - 1];
    const Counters *c = P.cnt;
    const uint32_t error = ld_volatile(&c->error), aside = ld_volatile(&c->aside), nq = ld_volatile(&c->queued);
    if (P.upd_mask && !aside && !(error & (ERR_SEQ_HALT | ERR_DEDUPE_FAILED | ERR_PENDING_OVERFLOW)))
      mark_queue(P, nq, nq, 0u, (blockIdx.x - blocks) * blockDim.x + threadIdx.x, (uint32_t)markers * blockDim.x);
    return;
  }
  const MapFrame &F = bd->f[m0 + blockIdx.y];
  Counters *cnt = F.cnt;
  // a de-duplication that did not complete leaves the frame out, and so does
  // a sequence halted by an earlier frame: the octree is not touched
  if (ld_volatile(&cnt->error) & (ERR_DEDUPE_FAILED | ERR_SEQ_HALT)) return;
  const uint32_t cands = ld_volatile(&cnt->cands);
  const int lane = threadIdx.x & 31;
  for (uint32_t j0 = blockIdx.x * blockDim.x + threadIdx.x - lane; j0 < cands; j0 += blocks * blockDim.x) {
    uint32_t levels = 0;
    if (j0 + lane < cands) {
      const uint4 c = F.cand[j0 + lane];
      bool created = false;
      uint32_t path[DESCENT_MAX];
      int np = 0;
      levels = insert_descend(F, c.z, c.x & 0xFFFFu, c.x >> 16, c.y & 0xFFFFu, c.y >> 16, cnt, &created, path, &np);
      if (created) stamp_path(F, path, np);
    }
    __syncwarp();
    // octree levels probed, when the stage profile is on (the algorithmic
    // bytes of the insert: 16 B per level -- the node's leaf and child slots,
    // the leaf's frame stamp and its queue entry, 4 B each)
    if (F.count_levels) {
      levels = __reduce_add_sync(0xffffffffu, levels);
      if (lane == 0) atomicAdd(&cnt->levels, levels);
    }
  }
}

// Enough blocks for a list as long as the image (every pixel its own cell),
// but no more than are resident at once.
void launch_insert(const BatchDesc *d_batch, uint32_t npix, int sm_count, cudaStream_t s, int block, int m0, int nmaps,
                   bool pdl, bool chained) {
  if (!npix || nmaps < 1) return;
  if (block < 64 || block > 1024 || block % 32) block = 256;
  const int resident = std::max(1, 1536 / block) * sm_count;
  const int blocks = std::max(1, std::min((int)((npix + block - 1) / block), resident / nmaps));
  note_launch();
  const int markers = chained ? MARK_BLOCKS : 0;
  launch_pdl(pdl, k_insert, dim3(blocks + markers, nmaps), dim3(block), 0, s, d_batch, m0, markers);
}

// ------------------------------------------------- pending leaf order -----

__global__ void k_pending_keys(const PendingLeaf *pend, int npend, uint64_t *keys) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= npend) return;
  keys[i] = pend[i].first_pixel;
}

size_t pending_sort_bytes(int n) { return argsort_temp_bytes((uint32_t)std::max(n, 0)); }

cudaError_t sort_pending(const PendingLeaf *pend, int npend, uint64_t *keys, uint64_t *keys_sorted, uint32_t *order,
                         void *tmp, size_t tmp_bytes, int end_bit, cudaStream_t s) {
  if (npend <= 0) return cudaSuccess;
  note_launch();
  k_pending_keys<<<(npend + 255) / 256, 256, 0, s>>>(pend, npend, keys);
  unsigned launches = 0;
  const cudaError_t e = argsort_u64(keys, (uint32_t)npend, end_bit, keys_sorted, order, tmp, tmp_bytes, s, &launches);
  note_launch(launches);
  return e;
}

// Leaf index = leaves_before + rank of first pixel; indices past the pool are
// stored in the tree but get no leaf record, like addLeaf's overflow
// (traversal_functions.cpp:201-210).
__device__ __forceinline__ void finalize_one(const PendingLeaf &p, uint32_t idx, uint32_t leaves_max, uint32_t *tree,
                                             ushort4 *leaf, uint32_t frame, uint32_t *stamp, uint32_t *queue,
                                             Counters *cnt) {
  tree[p.slot] = idx;
  if (idx < leaves_max) {
    leaf[idx] = p.pos;
    queue_leaf(idx, frame, stamp, queue, cnt);
  }
}

// A new leaf of rank r in its frame: index leaves_before + r, queued at
// position q0 + r after the q0 bricks the insert queued (a pending leaf is
// never on the insert's queue), so no atomics; the frame's queue length
// becomes q0 + the number of leaves placed.
__device__ __forceinline__ void finalize_new(const PendingLeaf &p, uint32_t idx, uint32_t qpos, uint32_t leaves_max,
                                             uint32_t *tree, ushort4 *leaf, uint32_t frame, uint32_t *stamp,
                                             uint32_t *queue) {
  tree[p.slot] = idx;
  if (idx < leaves_max) {
    leaf[idx] = p.pos;
    stamp[idx] = frame;
    queue[qpos] = idx;
  }
}

__global__ void k_finalize(const PendingLeaf *pend, const uint32_t *order, int npend, uint32_t leaves_before,
                           uint32_t leaves_max, uint32_t *tree, ushort4 *leaf, uint32_t frame, uint32_t *stamp,
                           uint32_t *queue, Counters *cnt) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npend) return;
  finalize_one(pend[order[j]], leaves_before + (uint32_t)j, leaves_max, tree, leaf, frame, stamp, queue, cnt);
}

void launch_finalize(const PendingLeaf *pend, const uint32_t *order, int npend, uint32_t leaves_before,
                     uint32_t leaves_max, uint32_t *tree, ushort4 *leaf, uint32_t frame, uint32_t *stamp,
                     uint32_t *queue, Counters *cnt, cudaStream_t s) {
  if (npend <= 0) return;
  note_launch();
  k_finalize<<<(npend + 255) / 256, 256, 0, s>>>(pend, order, npend, leaves_before, leaves_max, tree, leaf, frame,
                                                 stamp, queue, cnt);
}

// parent = finest ancestor leaf that existed when this leaf was created: the
// reference records the last leaf met on the descent (`pl`,
// traversal_functions.cpp:327-333, 376-379); leaves of this frame exist in
// index order, so that is the finest ancestor with a smaller index.
__device__ __forceinline__ uint32_t parent_of(uint32_t idx, uint32_t leaves_max, const uint32_t *tree, uint32_t n,
                                              const ushort4 &p) {
  const uint32_t edge = (uint32_t)p.w * BL;
  uint32_t ox = 0, oy = 0, oz = 0, half = n >> 1, branch = 0, pl = BRANCHINIT;
  while (half > edge) {
    uint32_t co = (p.x >= ox + half) * 1u + (p.y >= oy + half) * 2u + (p.z >= oz + half) * 4u;
    uint32_t l = tree[branch + co];
    if (l < leaves_max && l < idx) pl = l;
    branch = tree[branch + co + 8];
    if (branch >= PENDING) break;  // no child branch (cannot happen for a placed leaf)
    ox += half * ((co & 1) != 0);
    oy += half * ((co & 2) != 0);
    oz += half * ((co & 4) != 0);
    half >>= 1;
  }
  return pl;
}

__global__ void k_parents(int npend, uint32_t leaves_before, uint32_t leaves_max, const uint32_t *tree, uint32_t n,
                          const ushort4 *leaf, uint32_t *parent) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= npend) return;
  const uint32_t idx = leaves_before + (uint32_t)j;
  if (idx >= leaves_max) return;
  parent[idx] = parent_of(idx, leaves_max, tree, n, leaf[idx]);
}

// Parents of the leaves the finalisation of each frame of the descriptor
// placed: blocks PARENT_BLOCKS per frame, striding over its new leaves.  A
// parent is the finest ancestor with a smaller index, so it can be found any
// time after the leaf is placed; off the chain of frames (the next frame's
// insert does not wait for it).  Frames that placed nothing are skipped.
constexpr int PARENT_BLOCKS = 4, PARENT_THREADS = 256;

__global__ void __launch_bounds__(PARENT_THREADS) k_parents_frames(const BatchDesc *__restrict__ bd, int m0) {
  pdl_enter();
  const MapFrame &F = bd->f[m0 + blockIdx.x / PARENT_BLOCKS];
  const Counters *cnt = F.cnt;
  if (ld_volatile(&cnt->error) & (ERR_DEDUPE_FAILED | ERR_PENDING_OVERFLOW | ERR_SEQ_HALT)) return;
  const uint32_t npend = ld_volatile(&cnt->pending);
  const uint32_t leaves_before = F.chain ? ld_volatile(&cnt->leaves_base) : F.leaves_before;
  const uint32_t stride = PARENT_BLOCKS * PARENT_THREADS;
  for (uint32_t j = (blockIdx.x % PARENT_BLOCKS) * PARENT_THREADS + threadIdx.x; j < npend; j += stride) {
    const uint32_t idx = leaves_before + j;
    if (idx >= F.leaves_max) break;
    F.parent[idx] = parent_of(idx, F.leaves_max, F.tree, F.n, F.leaf[idx]);
  }
}

void launch_parents_frames(const BatchDesc *d_batch, int nframes, cudaStream_t s, int m0, bool pdl) {
  if (nframes < 1) return;
  note_launch();
  launch_pdl(pdl, k_parents_frames, dim3(nframes * PARENT_BLOCKS), dim3(PARENT_THREADS), 0, s, d_batch, m0);
}

// The whole frame's pending leaves in one block.  A leaf's creation rank is
// the number of pending leaves with a smaller first pixel; first pixels are
// distinct (a pixel creates at most one leaf), so the rank is a prefix count
// over a bitmap of the image's pixels held in shared memory.  Then indices,
// the leaf table and the parents.
constexpr int FIN_THREADS = 1024;
constexpr size_t FIN_SMEM_MAX = 200 * 1024;
constexpr int FIN_FEW = 1024;  // new leaves ranked by direct count (the dynamic shared memory holds >= 1024 words)

// One block per map of the batch; the pending count is read on the device
// (nothing is done after an allocation error, which the host reports).
// A frame of a sequence hands the next frame its branch count and leaf base,
// or halts it (and so every later frame) when this frame must grow the
// volume, failed or was halted itself: the host runs those frames again after
// the growth, or reports the failure.
__device__ __forceinline__ void chain_next(const MapFrame &F, Counters *cnt, uint32_t leaves_before, bool halt) {
  Counters *nx = F.next_cnt;
  if (!nx) return;
  nx->branches_used = ld_volatile(&cnt->branches_used);
  nx->leaves_base = leaves_before + ld_volatile(&cnt->pending);
  if (halt) atomicOr(&nx->error, ERR_SEQ_HALT);
}

__global__ void __launch_bounds__(FIN_THREADS) k_finalize_bitmap(const BatchDesc *__restrict__ bd, int m0) {
  extern __shared__ uint32_t fin_smem[];
  // (the next frame's insert is scheduled once this has started: it overlaps
  // this kernel, not the insert before it)
  pdl_wait();
  pdl_trigger();
  const MapFrame &F = bd->f[m0 + blockIdx.x];
  Counters *cnt = F.cnt;
  if (F.chain || F.next_cnt) {
    // a sequence's frame: everything it reads of the counters was written by
    // earlier kernels (its own insert, the previous finalisation)
    if (ld_volatile(&cnt->error) & (ERR_SEQ_HALT | ERR_DEDUPE_FAILED | ERR_PENDING_OVERFLOW)) {
      if (threadIdx.x == 0) chain_next(F, cnt, F.chain ? ld_volatile(&cnt->leaves_base) : F.leaves_before, true);
      return;
    }
  }
  // After a de-duplication error nothing was inserted.  After an insert whose
  // wait gave up (ERR_SPIN_TIMEOUT) the pending leaves recorded before it are
  // complete records and are placed, so that no octree slot keeps a pending
  // mark; the frame's update is skipped (ERR_FRAME_FAILED).
  if (cnt->error & (ERR_DEDUPE_FAILED | ERR_PENDING_OVERFLOW)) return;
  const int npend = (int)cnt->pending;
  const uint32_t q0 = cnt->queued;  // the insert's queue
  const uint32_t branches_used = cnt->branches_used;
  const PendingLeaf *pend = F.pend;
  const uint32_t leaves_before = F.chain ? ld_volatile(&cnt->leaves_base) : F.leaves_before;
  const uint32_t npix = F.npix, leaves_max = F.leaves_max, frame = F.frame;
  // the new leaves that fit the pool (indices below leaves_max) are queued
  const uint32_t nplaced = leaves_before < leaves_max ? min((uint32_t)npend, leaves_max - leaves_before) : 0u;
  const int t = threadIdx.x;
  // Whether the deferred update takes the frame (not when it failed or the
  // volume must grow first: the host handles those), decided by one thread
  // for the block (the confidence network, on another stream, may set its
  // error word meanwhile).  A map in one part marks its queue at once: the
  // marks need no leaf of this frame placed, so their atomics overlap the
  // ranking below; a part of a sharded map needs the new leaves' positions
  // and marks after it.
  __shared__ int aside_flag;
  if (t == 0) aside_flag = fuse_deferred(F) ? 1 : 0;
  __syncthreads();
  const bool stand_aside = aside_flag != 0;
  // (a frame with another after it in its chain is marked beside that one's insert)
  const bool mark = F.upd_mask && !stand_aside && !F.next_cnt;
  if (mark && F.shards <= 1) mark_queue(F, q0, q0 + nplaced, leaves_before, t, FIN_THREADS);
  uint32_t *rank = F.rank, *tree = F.tree, *stamp = F.stamp, *queue = F.queue;
  ushort4 *leaf = F.leaf;
  const uint32_t nwords = (npix + 31) / 32;
  uint32_t *bitmap = fin_smem;
  uint32_t *chunk_base = fin_smem + nwords;  // [FIN_THREADS]
  const uint32_t chunk = (nwords + FIN_THREADS - 1) / FIN_THREADS;
  if (npend <= FIN_FEW) {
    // few new leaves (the usual frame): a leaf's rank counted directly over
    // the others' first pixels in shared memory, without the image bitmap
    uint32_t *fp = fin_smem;
    for (int j = t; j < npend; j += FIN_THREADS) fp[j] = pend[j].first_pixel;
    __syncthreads();
    for (int j = t; j < npend; j += FIN_THREADS) {
      const uint32_t mine_fp = fp[j];
      uint32_t r = 0;
      for (int i = 0; i < npend; i++) r += fp[i] < mine_fp ? 1u : 0u;
      rank[j] = r;
      finalize_new(pend[j], leaves_before + r, q0 + r, leaves_max, tree, leaf, frame, stamp, queue);
    }
  } else {
    for (uint32_t w = t; w < nwords; w += FIN_THREADS) bitmap[w] = 0;
    __syncthreads();
    for (int j = t; j < npend; j += FIN_THREADS) {
      const uint32_t fp = pend[j].first_pixel;
      atomicOr(&bitmap[fp >> 5], 1u << (fp & 31));
    }
    __syncthreads();
    // the image bitmap of first pixels; exclusive prefix of the per-thread
    // chunk counts
    uint32_t mine = 0;
    const uint32_t w0 = (uint32_t)t * chunk, w1 = min(nwords, w0 + chunk);
    for (uint32_t w = w0; w < w1; w++) mine += __popc(bitmap[w]);
    using Scan = cub::BlockScan<uint32_t, FIN_THREADS>;
    __shared__ typename Scan::TempStorage scan_tmp;
    uint32_t before = 0;
    Scan(scan_tmp).ExclusiveSum(mine, before);
    chunk_base[t] = before;
    __syncthreads();
    for (int j = t; j < npend; j += FIN_THREADS) {
      const PendingLeaf p = pend[j];
      const uint32_t w = p.first_pixel >> 5, c = w / chunk;
      uint32_t r = chunk_base[c];
      for (uint32_t k = c * chunk; k < w; k++) r += __popc(bitmap[k]);
      r += __popc(bitmap[w] & ((1u << (p.first_pixel & 31)) - 1u));
      rank[j] = r;
      finalize_new(p, leaves_before + r, q0 + r, leaves_max, tree, leaf, frame, stamp, queue);
    }
  }
  // (the new leaves' parents: k_parents_frames, after this kernel)
  if (mark && F.shards > 1) {
    __syncthreads();  // the new leaves' positions
    mark_queue(F, q0, q0 + nplaced, leaves_before, t, FIN_THREADS);
  }
  if (t == 0) {
    cnt->queued = q0 + nplaced;
    cnt->aside = stand_aside ? 1u : 0u;
    Counters *nx = F.next_cnt;
    if (nx) {
      // the next frame of a sequence starts from this one's counts
      nx->branches_used = branches_used;
      nx->leaves_base = leaves_before + (uint32_t)npend;
      if (stand_aside) atomicOr(&nx->error, ERR_SEQ_HALT);
    }
  }
}

bool finalize_small_fits(uint32_t npix) {
  return sizeof(uint32_t) * (((size_t)npix + 31) / 32 + FIN_THREADS) <= FIN_SMEM_MAX;
}

bool finalize_small_prepare(int device) {
  static std::atomic<unsigned long long> attr_devices{0};
  const unsigned long long bit = 1ull << (device & 63);
  if (!(attr_devices.load() & bit)) {
    if (cudaFuncSetAttribute(k_finalize_bitmap, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FIN_SMEM_MAX) !=
        cudaSuccess)
      return false;
    attr_devices.fetch_or(bit);
  }
  return true;
}

bool launch_finalize_small(const BatchDesc *d_batch, int nmaps, uint32_t max_npix, int device, cudaStream_t s,
                           int m0, bool pdl) {
  const size_t smem = sizeof(uint32_t) * (((size_t)max_npix + 31) / 32 + FIN_THREADS);
  if (smem > FIN_SMEM_MAX || nmaps < 1) return false;
  if (!finalize_small_prepare(device)) return false;
  note_launch();
  return launch_pdl(pdl, k_finalize_bitmap, dim3(nmaps), dim3(FIN_THREADS), smem, s, d_batch, m0) == cudaSuccess;
}

void launch_parents(int npend, uint32_t leaves_before, uint32_t leaves_max, const uint32_t *tree, uint32_t n,
                    const ushort4 *leaf, uint32_t *parent, cudaStream_t s) {
  if (npend <= 0) return;
  note_launch();
  k_parents<<<(npend + 255) / 256, 256, 0, s>>>(npend, leaves_before, leaves_max, tree, n, leaf, parent);
}

// ---------------------------------------------------------------- grow ----

__global__ void k_shift_branches(uint32_t *tree, uint32_t used, uint32_t shift) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= used) return;
  if ((i & 15) >= 8 && tree[i] != BRANCHINIT) tree[i] += shift;
}

void launch_shift_branches(uint32_t *tree, uint32_t used, uint32_t shift, cudaStream_t s) {
  if (!used) return;
  note_launch();
  k_shift_branches<<<(used + 255) / 256, 256, 0, s>>>(tree, used, shift);
}

__global__ void k_shift_leaves(ushort4 *leaf, uint32_t n, ushort3 add) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  ushort4 p = leaf[i];
  p.x = (uint16_t)(p.x + add.x);
  p.y = (uint16_t)(p.y + add.y);
  p.z = (uint16_t)(p.z + add.z);
  leaf[i] = p;
}

void launch_shift_leaves(ushort4 *leaf, uint32_t n, ushort3 add, cudaStream_t s) {
  if (!n) return;
  note_launch();
  k_shift_leaves<<<(n + 255) / 256, 256, 0, s>>>(leaf, n, add);
}

__global__ void k_fill(uint32_t *p, size_t n, uint32_t v) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) p[i] = v;
}

void launch_fill(uint32_t *p, size_t n, uint32_t v, cudaStream_t s) {
  if (!n) return;
  size_t blocks = (n + 255) / 256;
  if (blocks > 148 * 32) blocks = 148 * 32;
  note_launch();
  k_fill<<<(unsigned)blocks, 256, 0, s>>>(p, n, v);
}

// Load this file's kernels now (modules load lazily on first launch, which
// would otherwise land inside the first frame that needs a kernel).
cudaError_t prewarm_alloc_kernels() {
  const void *fns[] = {(const void *)k_first_bbox, (const void *)k_dedupe<DD_ROWS_SHORT>,
                       (const void *)k_dedupe_one<DD_ROWS_SHORT>, (const void *)k_dedupe_one<DD_ROWS_LOW>,
                       (const void *)k_dedupe_one<DD_ROWS_TALL>,
                       (const void *)k_dedupe<DD_ROWS_LOW>,
                       (const void *)k_dedupe<DD_ROWS_TALL>, (const void *)k_insert,
                       (const void *)k_pending_keys, (const void *)k_finalize, (const void *)k_parents, (const void *)k_parents_frames,
                       (const void *)k_finalize_bitmap, (const void *)k_shift_branches,
                       (const void *)k_shift_leaves, (const void *)k_fill};
  for (const void *f : fns) {
    cudaFuncAttributes a;
    cudaError_t e = cudaFuncGetAttributes(&a, f);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace ffb
