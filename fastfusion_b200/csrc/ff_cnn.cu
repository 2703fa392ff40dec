// Learned per-pixel confidence weight: a 3-layer 5x5 CNN (16 channels) with
// BF16 weights and activations and FP32 accumulation, its training kernels
// (backward of every layer, MSE loss, Adam), the input features, and a
// raycaster of the fused volume that gives the training targets.
//
// There is no counterpart in the reference: its fusion weight is the fixed
// distance ramp of update_functions.cpp:1187-1444.  The learned weight
// multiplies that ramp's weight increment per pixel; with no network set the
// update is the reference's, bit for bit.
//
// Layout in HBM (n images of W x H, pixel-major, channels innermost):
//   features  bf16 [n][H][W][8]   depth (m), normal (x, y, z), valid, 0, 0, 0
//   a1, a2    bf16 [n][H][W][16]  post-ReLU activations of layers 1 and 2
//   pred      f32  [n][H][W]      layer 3 output: predicted |depth residual| in cm
//   params    bf16 [8833]         W1[16][5][25] b1[16] W2[16][16][25] b2[16] W3[1][16][25] b3[1]
// Convolutions are 'same' 5x5 correlations with zero padding per image.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <mutex>

#include "ff_common.cuh"
#include "ff_kernels.h"

namespace ffb {

constexpr int CNN_HID = 16;
constexpr int CNN_IN = 5;
constexpr int CNN_IN_STRIDE = 8;
constexpr int TAPS = 25;
constexpr int P_W1 = 0, P_B1 = P_W1 + CNN_HID * CNN_IN * TAPS, P_W2 = P_B1 + CNN_HID,
              P_B2 = P_W2 + CNN_HID * CNN_HID * TAPS, P_W3 = P_B2 + CNN_HID, P_B3 = P_W3 + CNN_HID * TAPS,
              P_TOTAL = P_B3 + 1;
static_assert(P_TOTAL == CNN_PARAMS && CNN_HID == CNN_HIDDEN && CNN_IN_STRIDE == CNN_FEAT_CH, "parameter layout");

enum ConvMode { CONV_RELU_BF16 = 0, CONV_F32 = 1, CONV_CONF = 2 };

// ------------------------------------------------ tensor-core convolution
//
// The forward layers as streamed implicit GEMMs on the 5th-generation tensor
// cores.  Output rows come in groups of four ("quads"): for input row t of the
// eight that a quad reads and for kernel column kx, one tcgen05.mma (M = 128
// pixels, K = 16, BF16, FP32 accumulator in tensor memory) adds
//   D[pixel p][16 j + co] += sum over ci of x[t][p + kx][ci] * w[co][ci][t - j][kx]
// for all output rows j at once that have row t in their window (one to four of
// them: N = 16 to 64; a row's very first product is an MMA of its own, which
// sets its columns).  The shift kx is the start address of the A descriptor; the
// rows of a t are a window into one strip of five column blocks per kx, ky from
// the last to the first, so they are the start address of B's.
// Why: an M = 128 MMA reads (128 + N) x 32 bytes of operands from shared
// memory, 128 bytes a cycle.  One MMA per tap with N = 16 takes 25 x 36 = 900
// cycles a row; a quad takes 43 MMAs of 36 to 48, 450 a row.  Only products of an
// output's own window enter its sum, so that an infinite activation stays within
// the outputs that see it; and every output is the sum of its taps in raster
// order (K = 16 at a time), the order the activations' BF16 rounding is defined by.
//
// The one-channel layer packs the four rows' columns into one N = 16, the smallest:
// 40 MMAs of 36 a quad, 360 a row, the strips with zeros for the rows that row t
// is no part of, which add nothing as long as the input is finite.  Loader warps note
// where it is not, and a quad that reads such values takes its rows one by one
// (100 MMAs).
//
// Operands: K-major, unswizzled canonical layout (8 x 16-byte core matrices,
// pixels 16 bytes apart, 8-pixel groups 128 (SBO), the two 8-channel halves
// of K one plane apart (LBO); 8 channels: the halves are two neighbouring
// pixels, 16 bytes apart, and serve two kx).
//
// A block streams down its strip: loader warps bring quads of input rows into a
// ring in shared memory (each row once: only the 4 halo rows at a block's
// ends are read twice), issuing threads run the MMAs of a quad as soon as
// its two input quads are there, and epilogue warps empty the accumulators.
// Four issuers, each with an accumulator of its own, since the MMAs of one
// accumulator wait for one another and one thread issues an MMA in about 80
// cycles.  The quads of all strips of all images are dealt out evenly, a
// block's share running over from one strip to the next.  All waits are
// bounded.
//
// Measured on four 640x480 images: layers 1, 2 and 3 take 25, 29 and 22 us, on one
// image 11, 14 and 10; layers 1 and 2 with N = 64 throughout (40 MMAs a quad, zeros
// for the rows out of reach, by which an infinite activation is multiplied) 26 and
// 29, and 12 and 15; layer 3 with 16 columns a row (N = 16 to 64) 25 and 13; a block
// per 128 x 8 pixels with one MMA per tap, N = 16, 34, 50 and 44, and 13, 19 and 17.
constexpr int TC_WAIT_LIMIT = 1 << 24;  // polls (a wait takes microseconds: one that gives up means a fault, not a slow device)
constexpr int CQ_OUT = 128;      // output pixels of a strip
constexpr int CQ_PX = 136;       // input pixels of a ring row: 128 + 4, whole 128-byte core matrices
constexpr int CQ_PLANE = CQ_PX * 16;  // bytes of one 8-channel plane of an input row
constexpr int CQ_SLOTS = 5;      // quads of input rows in the ring
constexpr int CQ_EPI_WARPS = 8, CQ_LOAD_WARPS = 8, CQ_MMA_WARPS = 4;
constexpr int CQ_THREADS = 32 * (CQ_EPI_WARPS + CQ_LOAD_WARPS + CQ_MMA_WARPS);

// C: input channels (8 or 16)
template <int C>
struct CqIn {
  static constexpr int PLANES = C / 8;
  static constexpr int ROW = PLANES * CQ_PLANE;
  static constexpr int QUAD = 4 * ROW;
  static constexpr int NKX = C == 8 ? 3 : 5;  // MMAs per t
};
constexpr int CQ_ACC = 4 * 16;     // columns of an accumulator
constexpr int CQ_COLS = CQ_MMA_WARPS * CQ_ACC;
// columns of a kx's weight strip: a block of 16 per ky; one output channel: 3 zeros,
// a column per ky, zeros
template <int COUT>
__host__ __device__ constexpr int cq_strip() {
  return COUT == 1 ? 24 : 5 * 16;
}
template <int C, int COUT>
__host__ __device__ constexpr int cq_weight_bytes() {
  return CqIn<C>::NKX * cq_strip<COUT>() * 32;
}
template <int C, int COUT>
constexpr size_t cq_smem_bytes() {
  return (size_t)CQ_SLOTS * CqIn<C>::QUAD + cq_weight_bytes<C, COUT>() + 256;
}

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, no swizzle (sm_100 version 1)
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}

// instruction descriptor: D FP32, A and B BF16, both K-major, M = 128
__host__ __device__ constexpr uint32_t tc_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24);
}

// TMA tile loads and a bulk copy, completing on an mbarrier (transaction bytes)
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *m, int c0, int c1, int c2, int c3,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *m, int c0, int c1, int c2, int c3,
                                            int c4, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
      "%6}], [%7];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(bar)
      : "memory");
}
__device__ __forceinline__ uint32_t mbar_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok = 0;
  for (int it = 0; it < TC_WAIT_LIMIT && !ok; it++) {
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
  }
  return ok;
}

// The three BF16 parts of v (bit patterns in the upper halves): v = hi + mid +
// lo, exactly down to 2^-110 (below that the low part leaves BF16's range); an
// infinity or a NaN stays in hi alone.
__device__ __forceinline__ void split3_bf16(float v, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
  hi = __float_as_uint(v) & 0xFFFF0000u;
  float r = v - __uint_as_float(hi);
  r = r == r ? r : 0.0f;
  mid = __float_as_uint(r) & 0xFFFF0000u;
  lo = __float_as_uint(r - __uint_as_float(mid));
}
// the upper halves of a and b as two BF16 words, a first
__device__ __forceinline__ uint32_t pack_hi(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr));
}
__device__ __forceinline__ void tmem_ld1(uint32_t addr, uint32_t &v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(addr));
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void tc_commit(uint64_t *bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}
// A bounded wait; one that gives up sets *stop, on which every later wait of
// the block gives up at once.
__device__ __forceinline__ bool tc_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *stop) {
  const uint32_t addr = smem_addr(bar);
  for (int it = 0; it < TC_WAIT_LIMIT; it++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*stop) return false;
  }
  *stop = 1u;
  return false;
}
__device__ __forceinline__ void tc_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// A block's share of the output quads: segments of consecutive quads of one
// strip.
struct CqSeg {
  int64_t r, end;  // position in the quad space, strip after strip; the share's end
  int img, x0, y0, len;  // first output pixel and row, quads
};
__device__ __forceinline__ void cq_seg(CqSeg &s, int quads, int strips) {
  const int64_t strip = s.r / quads;
  const int first = (int)(s.r - strip * quads);
  s.img = (int)(strip / strips);
  s.x0 = (int)(strip % strips) * CQ_OUT;
  s.y0 = 4 * first;
  s.len = (int)min((int64_t)(quads - first), s.end - s.r);
}

// Pixel (x, y) of image img as loaded: C BF16 channels, zero outside the image.
template <int C>
struct CqPx {
  uint4 v[C / 8];
};
template <int C>
__device__ __forceinline__ void cq_load_px(CqPx<C> &p, const __nv_bfloat16 *__restrict__ in, int img, int x, int y,
                                           int W, int H) {
  const bool inside = x >= 0 && x < W && y >= 0 && y < H;
  const uint4 *q = reinterpret_cast<const uint4 *>(in) + (((int64_t)img * H + y) * W + x) * (C / 8);
#pragma unroll
  for (int k = 0; k < C / 8; k++) p.v[k] = inside ? __ldg(q + k) : make_uint4(0u, 0u, 0u, 0u);
}
// into position d of an input row (planes CQ_PLANE apart)
template <int C>
__device__ __forceinline__ void cq_store_px(const CqPx<C> &p, uint8_t *d) {
#pragma unroll
  for (int k = 0; k < C / 8; k++) *reinterpret_cast<uint4 *>(d + k * CQ_PLANE) = p.v[k];
}

// The largest of m's and a pixel's values as bit patterns (halves): from 0x7F80 on
// infinite, NaN or, behind a ReLU not met, negative.
template <int C>
__device__ __forceinline__ uint32_t cq_largest(const CqPx<C> &p, uint32_t m) {
#pragma unroll
  for (int k = 0; k < C / 8; k++) {
    m = __vimax3_u16x2(m, p.v[k].x, p.v[k].y);
    m = __vimax3_u16x2(m, p.v[k].z, p.v[k].w);
  }
  return m;
}

// Element (column n, k) of MMA column kxi's weight strip.  16 output channels:
// block i of a strip holds ky = 4 - i, its columns the output channels; one:
// column i holds ky = 7 - i (zero unless 0 .. 4).  k is the input channel (8
// channels: of pixel kx = 2 kxi, then of kx + 1).
template <int C, int COUT>
__device__ __forceinline__ __nv_bfloat16 cq_weight(const __nv_bfloat16 *__restrict__ w, int kxi, int n, int k) {
  constexpr int CIN = C == 8 ? CNN_IN : CNN_HID;
  const int co = COUT == 1 ? 0 : n & 15, ky = COUT == 1 ? 7 - n : 4 - (n >> 4);
  const int kx = C == 8 ? 2 * kxi + (k >> 3) : kxi, ci = k % C;
  if (ky < 0 || ky > 4 || kx > 4 || ci >= CIN) return __float2bfloat16_rn(0.0f);
  return __ldg(w + (co * CIN + ci) * TAPS + ky * 5 + kx);
}

template <int C, int COUT, int MODE>
__global__ void __launch_bounds__(CQ_THREADS, 1) k_conv_quads(const __nv_bfloat16 *__restrict__ in, int W, int H, int n_img,
                                                             const __nv_bfloat16 *__restrict__ w,
                                                             const __nv_bfloat16 *__restrict__ bias,
                                                             void *__restrict__ out, float inv_tau,
                                                             uint32_t *__restrict__ err, int err_stride) {
  using I = CqIn<C>;
  constexpr int STRIP = cq_strip<COUT>(), WBYTES = cq_weight_bytes<C, COUT>();
  extern __shared__ __align__(1024) uint8_t rsm[];
  uint8_t *ring = rsm;
  uint8_t *wsm = rsm + CQ_SLOTS * I::QUAD;  // [kx][k half][strip column][8] bf16
  uint64_t *full = reinterpret_cast<uint64_t *>(wsm + WBYTES);
  uint64_t *empty = full + CQ_SLOTS, *dfull = empty + CQ_SLOTS, *dempty = dfull + CQ_MMA_WARPS,
           *drain = dempty + CQ_MMA_WARPS;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile uint32_t *stop = tmem_slot + 1;
  // one output channel: how an accumulator holds its rows (1: a column each, 16:
  // 16 columns each), and whether a loader warp's share of a slot has values that
  // are not finite
  volatile uint32_t *row_cols = tmem_slot + 2;
  volatile uint8_t *not_finite = reinterpret_cast<volatile uint8_t *>(tmem_slot + 2 + CQ_MMA_WARPS);
  static_assert((2 * CQ_SLOTS + 2 * CQ_MMA_WARPS + 2) * 8 + 4 * CQ_MMA_WARPS + CQ_SLOTS * CQ_LOAD_WARPS <= 256 &&
                    CQ_LOAD_WARPS == 8 && CQ_MMA_WARPS % 2 == 0,
                "barrier words");
  static_assert(I::QUAD % 128 == 0 && WBYTES % 16 == 0, "operand alignment");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool loader = warp >= CQ_EPI_WARPS && warp < CQ_EPI_WARPS + CQ_LOAD_WARPS;
  const int quads = (H + 3) / 4, strips = (W + CQ_OUT - 1) / CQ_OUT;
  const int64_t total = (int64_t)strips * n_img * quads;
  CqSeg seg;
  seg.r = total * blockIdx.x / gridDim.x;
  seg.end = total * (blockIdx.x + 1) / gridDim.x;

  // Loaders: a quad's 4 x 132 pixels over 256 threads, two rows of one pixel
  // column each and the last four columns by the first 16 (quad g of the
  // block's sequence goes to ring slot g % SLOTS); the next quad in flight
  // while they wait for its slot, the first of all while the block is set up.
  const int lt = tid - 32 * CQ_EPI_WARPS;
  const int lpx = lt & 127, lrow = (lt >> 7) * 2;
  CqSeg c = seg;
  int ci = 0;  // the segment's next input quad to fetch, 0 .. len
  CqPx<C> p[3];
  auto fetch = [&] {
    if (c.r >= c.end) return;
    const int gy = c.y0 - 2 + 4 * ci, gx = c.x0 - 2;
    cq_load_px<C>(p[0], in, c.img, gx + lpx, gy + lrow, W, H);
    cq_load_px<C>(p[1], in, c.img, gx + lpx, gy + lrow + 1, W, H);
    if (lt < 16) cq_load_px<C>(p[2], in, c.img, gx + 128 + (lt & 3), gy + (lt >> 2), W, H);
    if (++ci < c.len + 1) return;
    c.r += c.len;
    ci = 0;
    if (c.r < c.end) cq_seg(c, quads, strips);
  };
  if (loader) {
    if (c.r < c.end) cq_seg(c, quads, strips);
    fetch();
  } else {
    // (a thread's weights in flight together)
    constexpr int SETUP = CQ_THREADS - 32 * CQ_LOAD_WARPS, WN = WBYTES / 2, PER = (WN + SETUP - 1) / SETUP;
    const int t = warp < CQ_EPI_WARPS ? tid : tid - 32 * CQ_LOAD_WARPS;
#pragma unroll 8
    for (int k = 0; k < PER; k++) {
      const int i = t + k * SETUP, r = (i >> 3) / STRIP;
      if (i < WN)
        reinterpret_cast<__nv_bfloat16 *>(wsm)[i] =
            cq_weight<C, COUT>(w, r >> 1, (i >> 3) % STRIP, (r & 1) * 8 + (i & 7));
    }
    // (the ring's pixels 132 .. 135 are never written: the 8-channel layer's
    // last tap pair reads pixel 132 against zero weights)
    if constexpr (C == 8)
      for (int i = t; i < 4 * CQ_SLOTS * 4; i += SETUP)
        *reinterpret_cast<uint4 *>(ring + (i >> 2) * I::ROW + (132 + (i & 3)) * 16) = make_uint4(0u, 0u, 0u, 0u);
    if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                   "r"(CQ_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 32) {
      auto init = [](uint64_t *b, uint32_t n) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(n));
      };
      for (int k = 0; k < CQ_SLOTS; k++) init(full + k, CQ_LOAD_WARPS), init(empty + k, CQ_MMA_WARPS);
      for (int k = 0; k < CQ_MMA_WARPS; k++) init(dfull + k, COUT == 1 ? 2 : 1), init(dempty + k, CQ_EPI_WARPS);
      init(drain, CQ_MMA_WARPS);
      *stop = 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (loader) {
    // input quads of the whole share: its output quads, and the halo of each segment
    const int64_t segs = seg.r < seg.end ? (seg.end - 1) / quads - seg.r / quads + 1 : 0;
    const uint32_t count = (uint32_t)(seg.end - seg.r + segs);
    uint32_t sl = 0, par = 1;  // ring slot; parity of the wait for it (at once in the first turn)
    for (uint32_t g = 0; g < count; g++) {
      // (the warp stops as one: its lanes meet below)
      if (!__all_sync(0xffffffffu, tc_wait(empty + sl, par, stop))) break;
      uint8_t *d = ring + sl * I::QUAD;
      cq_store_px<C>(p[0], d + lrow * I::ROW + lpx * 16);
      cq_store_px<C>(p[1], d + (lrow + 1) * I::ROW + lpx * 16);
      if (lt < 16) cq_store_px<C>(p[2], d + (lt >> 2) * I::ROW + (128 + (lt & 3)) * 16);
      if constexpr (COUT == 1) {
        uint32_t u = cq_largest<C>(p[1], cq_largest<C>(p[0], 0u));
        if (lt < 16) u = cq_largest<C>(p[2], u);
        const bool any = __any_sync(0xffffffffu, (u & 0xFFFFu) >= 0x7F80u || u >= 0x7F800000u);
        if (lane == 0) not_finite[sl * CQ_LOAD_WARPS + warp - CQ_EPI_WARPS] = any ? 1 : 0;
      }
      __syncwarp();
      if (lane == 0) tc_arrive(full + sl);
      if (++sl == CQ_SLOTS) sl = 0, par ^= 1;
      fetch();
    }
  } else if (warp >= CQ_EPI_WARPS) {
    if (lane == 0) {
      // MMAs: of every segment, issuer m takes output quads m, m + 4, ... into
      // its own accumulator.  Quad k reads input quads k and k + 1, there
      // when the second is (the loaders take them in order).  Every issuer
      // releases every input quad once, in order: by a commit after its last
      // output quad that reads it, or, reading none of it, after it has
      // passed; so no phase of a slot is missed.
      const uint32_t m = (uint32_t)(warp - CQ_EPI_WARPS - CQ_LOAD_WARPS);
      const uint32_t rbase = smem_addr(ring), wbase = smem_addr(wsm), acc = tmem + m * CQ_ACC;
      uint32_t g = 0, dpar = 1;  // the segment's first input quad; parity of the wait for the accumulator
      bool ok = true;
      auto wait_full = [&](uint32_t gi) { return tc_wait(full + gi % CQ_SLOTS, (gi / CQ_SLOTS) & 1, stop); };
      while (seg.r < seg.end && ok) {
        cq_seg(seg, quads, strips);
        const uint32_t len = (uint32_t)seg.len;
        uint32_t q = 0;  // the segment's next input quad to release
        for (uint32_t k = m;; k += CQ_MMA_WARPS) {
          const uint32_t upto = k < len ? k : len + 1;
          for (; q < upto && ok; q++) {
            ok = wait_full(g + q);
            if (ok) tc_arrive(empty + (g + q) % CQ_SLOTS);
          }
          if (k >= len || !ok) break;
          const uint32_t gi = g + k;
          ok = wait_full(gi + 1) && tc_wait(dempty + m, dpar, stop);
          if (!ok) break;
          dpar ^= 1;
          // the loaders' stores, acquired through their barrier, ordered
          // before the tensor core's reads
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t s0 = rbase + gi % CQ_SLOTS * I::QUAD, s1 = rbase + (gi + 1) % CQ_SLOTS * I::QUAD;
          constexpr int KXS = C == 8 ? 32 : 16, LBO = C == 8 ? 16 : CQ_PLANE;
          if constexpr (COUT == 1) {
            const volatile uint32_t *f0 =
                reinterpret_cast<const volatile uint32_t *>(not_finite + gi % CQ_SLOTS * CQ_LOAD_WARPS);
            const volatile uint32_t *f1 =
                reinterpret_cast<const volatile uint32_t *>(not_finite + (gi + 1) % CQ_SLOTS * CQ_LOAD_WARPS);
            const bool finite = !(f0[0] | f0[1] | f1[0] | f1[1]);
            row_cols[m] = finite ? 1u : 16u;
            if (finite) {
#pragma unroll
              for (int t = 0; t < 8; t++) {
                const uint32_t rb = (t < 4 ? s0 : s1) + (t & 3) * I::ROW;
                const uint32_t wb = wbase + (uint32_t)((7 - t) * 16);
#pragma unroll
                for (int kx = 0; kx < I::NKX; kx++)
                  tc_mma(acc, tc_desc(rb + kx * KXS, LBO, 128), tc_desc(wb + kx * STRIP * 32, STRIP * 16, 128),
                         tc_idesc(16), (kx || t) ? 1u : 0u);
              }
            } else {
              for (int i = 0; i < 4 * 5; i++) {
                const int j = i / 5, ky = i % 5, t = j + ky;
                const uint32_t rb = (t < 4 ? s0 : s1) + (t & 3) * I::ROW;
                const uint32_t wb = wbase + (uint32_t)((7 - ky) * 16);
#pragma unroll
                for (int kx = 0; kx < I::NKX; kx++)
                  tc_mma(acc + 16 * j, tc_desc(rb + kx * KXS, LBO, 128),
                         tc_desc(wb + kx * STRIP * 32, STRIP * 16, 128), tc_idesc(16), (kx || ky) ? 1u : 0u);
              }
            }
            tc_arrive(dfull + m);  // (row_cols, released to the epilogue: the phase takes this and the commit)
          } else {
#pragma unroll
            for (int t = 0; t < 8; t++) {
              // output rows j0 .. j1, from block 4 - t + j0 (ky = t - j0) on
              const int j0 = max(t - 4, 0), j1 = min(t, 3);
              const uint32_t rb = (t < 4 ? s0 : s1) + (t & 3) * I::ROW;
#pragma unroll
              for (int kx = 0; kx < I::NKX; kx++) {
                const uint64_t ad = tc_desc(rb + kx * KXS, LBO, 128);
                const uint32_t wk = wbase + (uint32_t)(kx * STRIP * 32);
                auto mma = [&](int j, int rows, uint32_t accumulate) {
                  tc_mma(acc + 16 * j, ad, tc_desc(wk + (uint32_t)((4 - t + j) * 256), STRIP * 16, 128),
                         tc_idesc(16 * rows), accumulate);
                };
                if (t < 4 && kx == 0) {  // row t's first product
                  if (t) mma(0, t, 1u);
                  mma(t, 1, 0u);
                } else {
                  mma(j0, j1 - j0 + 1, 1u);
                }
              }
            }
          }
          tc_commit(dfull + m);
          // the input quads this issuer's next output quad does not read
          for (; q <= k + 1; q++) tc_commit(empty + (g + q) % CQ_SLOTS);
        }
        g += len + 1;
        seg.r += seg.len;
      }
      // every MMA and commit done before the block's memory is given back
      tc_commit(drain);
      uint32_t never = 0u;
      tc_wait(drain, 0, &never);
    }
  } else {
    // Epilogue: two groups of four warps, two rows of every quad each; the
    // accumulators in turn, from the first in every segment
    const int quad = warp & 3, row0 = (warp >> 2) * 2;
    const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16);
    float b[COUT];
#pragma unroll
    for (int k = 0; k < COUT; k++) b[k] = __bfloat162float(__ldg(bias + k));
    uint32_t par = 0;  // bit d: parity of the next wait for accumulator d
    while (seg.r < seg.end) {
      cq_seg(seg, quads, strips);
      uint32_t d = 0;
      const int gx = seg.x0 + quad * 32 + lane;
      for (int i = 0; i < seg.len; i++) {
        const int gy = seg.y0 + 4 * i + row0;
        const size_t px0 = ((size_t)seg.img * H + gy) * W + gx;
        const bool inside[2] = {gx < W && gy < H, gx < W && gy + 1 < H};
        const bool ok = tc_wait(dfull + d, (par >> d) & 1, stop);
        __syncwarp();  // (the reads of tensor memory are by whole warps)
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t v[2][COUT];
        const uint32_t cols = COUT == 1 && row_cols[d] == 1u ? 1u : 16u;
        const uint32_t at = trow + d * CQ_ACC + row0 * cols;
        if constexpr (COUT == 1) {
          tmem_ld1(at, v[0][0]);
          tmem_ld1(at + cols, v[1][0]);
        } else {
          tmem_ld16(at, v[0]);
          tmem_ld16(at + 16, v[1]);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (lane == 0) tc_arrive(dempty + d);
        par ^= 1u << d;
        d = (d + 1) % CQ_MMA_WARPS;
#pragma unroll
        for (int r = 0; r < 2; r++) {
          if (!inside[r]) continue;
          const size_t px = px0 + (size_t)r * W;
          if constexpr (COUT == 1) {
            float a = __uint_as_float(v[r][0]) + b[0];
            if (!ok) a = __uint_as_float(0x7FC00000u);  // NaN: the accumulators were not read
            if (MODE == CONV_CONF) {
              // (1 - r/tau)^2 on [0, tau], 0 beyond: weight falls to exactly zero
              // for pixels whose predicted residual reaches tau
              const float f = fmaxf(1.0f - fmaxf(a, 0.0f) * inv_tau, 0.0f);
              a = ok ? f * f : a;
            }
            reinterpret_cast<float *>(out)[px] = a;
          } else {
            float a[16];
#pragma unroll
            for (int k = 0; k < 16; k++) a[k] = ok ? __uint_as_float(v[r][k]) + b[k] : __uint_as_float(0x7FC00000u);
            uint4 o[2];
            __nv_bfloat16 *ob = reinterpret_cast<__nv_bfloat16 *>(o);
#pragma unroll
            for (int k = 0; k < 16; k++) ob[k] = __float2bfloat16_rn(fmaxf(a[k], 0.0f));
            uint4 *dst = reinterpret_cast<uint4 *>(reinterpret_cast<__nv_bfloat16 *>(out) + px * 16);
            dst[0] = o[0];
            dst[1] = o[1];
          }
        }
        __syncwarp();
      }
      seg.r += seg.len;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (*stop && tid == 0 && err) {
    // every image the block had a share of
    const int64_t of_image = (int64_t)strips * quads;
    for (int64_t i = total * blockIdx.x / gridDim.x / of_image; i * of_image < total * (blockIdx.x + 1) / gridDim.x; i++)
      atomicOr(err + i * err_stride, ERR_SPIN_TIMEOUT);
  }
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(CQ_COLS));
}

// ------------------------------------------------ tensor-core input gradients
//
// The gradient of a layer's input, masked by the ReLU of the stored activation:
// a correlation of the FP32 output gradient with the layer's weights, transposed
// and flipped, as a streamed implicit GEMM.  Per output row of a strip, one
// tcgen05.mma (M = 128 input pixels, N = 80, K = 16) per kernel row ky and BF16
// part accumulates
//   D[input pixel s][kx * 16 + ci] = sum over ky, co of g[row + ky][s][co] * w[co][ci][4 - ky][4 - kx],
// all five kx side by side in N, and the epilogue adds
//   out[j][ci] = sum over kx of D[j + kx][kx * 16 + ci]
// across the lanes of a warp: a 32-pixel window belongs to each warp, so it
// gives 28 outputs, and the four windows of a strip start 28 pixels apart.
// Not as the forward layers: the gradient enters as three BF16 parts whose sum
// it is exactly (split3_bf16), so the MMAs count three times, and all kx in N
// take 15 of them a row where quads take 30; the fewer sums in the accumulator,
// which rounds toward zero, also keep the error below that of FP32
// multiply-adds (7.1e-8 and 8.5e-8 relative L2 for layers 3 and 2 against 64 bits;
// 8.8e-8 and 2.4e-7 with FP32, 1.4e-7 and 2.2e-7 as quads).  Layer 3's
// one-channel gradient has the three parts of its five rows ky in the K
// dimension: its ring holds an output row's operand, one MMA a row.
//
// Streaming as in the forward layers, two rows at a time: loader warps bring
// pairs of input rows into the ring, four issuers with an accumulator each take
// the output rows in turn, two groups of epilogue warps the rows of a pair.
//
// Measured on four 640x480 images: layers 3 and 2 take 43 and 74 us, bound by
// the epilogue's shuffles (64 per warp and row) and by the MMAs (15 a row,
// about 107 cycles each); FP32 multiply-adds on the CUDA cores 50 and 366 us.
constexpr int RC_OUT = 112;      // output pixels of a strip: 4 windows of 28
constexpr int RC_SLOTS = 6;      // pairs of input rows in the ring
constexpr int RC_PLANE = 128 * 16;  // bytes of one 8-channel plane of an input row
constexpr int RC_EPI_WARPS = 8, RC_LOAD_WARPS = 4, RC_MMA_WARPS = 4;
constexpr int RC_AHEAD = 2;      // pairs of input rows a loader has in flight
constexpr int RC_THREADS = 32 * (RC_EPI_WARPS + RC_LOAD_WARPS + RC_MMA_WARPS);
constexpr int RC_MIN_PAIRS = 2;  // pairs of output rows that are worth a block of their own

enum RcInput { RC_F32_16 = 0, RC_F32_1 = 1 };

template <int IN>
struct RcIn {
  static constexpr int PARTS = IN == RC_F32_16 ? 3 : 1;  // MMAs per kernel row
  static constexpr int ROW = 2 * PARTS * RC_PLANE;
  static constexpr int PAIR = 2 * ROW;
  static constexpr int KY = IN == RC_F32_1 ? 1 : 5;    // ring rows of an output row
  static constexpr int HALO = IN == RC_F32_1 ? 0 : 2;  // ring pairs of a segment beyond its output pairs
};
constexpr int RC_N = 80, RC_COLS = 512;  // columns of an accumulator (one per issuer), and allocated
static_assert(RC_MMA_WARPS * RC_N <= RC_COLS, "accumulators fit the allocation");
template <int IN>
constexpr size_t rc_smem_bytes() {
  return std::max<size_t>((size_t)RC_SLOTS * RcIn<IN>::PAIR + RcIn<IN>::KY * 2 * RC_N * 16 + 512,
                          114 * 1024);  // (one block per SM: all of tensor memory)
}

// A block's share of the output row pairs: segments of consecutive pairs of
// one strip (x0: its first output pixel).
struct RcSeg {
  int64_t r, end;  // position in the pair space, strip after strip; the share's end
  int img, x0, y0, len;  // first output row, pairs
};
__device__ __forceinline__ void rc_seg(RcSeg &s, int pairs, int strips) {
  const int64_t strip = s.r / pairs;
  const int first = (int)(s.r - strip * pairs);
  s.img = (int)(strip / strips);
  s.x0 = (int)(strip % strips) * RC_OUT;
  s.y0 = 2 * first;
  s.len = (int)min((int64_t)(pairs - first), s.end - s.r);
}

// One pixel's channels as loaded.
template <int IN>
struct RcPx {
  static constexpr int NV = IN == RC_F32_16 ? 4 : 2;
  uint4 v[NV];
};
// Pixel px = (y, x) of an image of H rows; a one-channel input: rows y - 2 .. y + 2 of
// its column (zero outside).
template <int IN>
__device__ __forceinline__ void rc_load_px(RcPx<IN> &p, const void *__restrict__ in, bool inside_x, int y, int H,
                                           int W, size_t px) {
#pragma unroll
  for (int k = 0; k < RcPx<IN>::NV; k++) p.v[k] = make_uint4(0u, 0u, 0u, 0u);
  if (!inside_x) return;
  if constexpr (IN == RC_F32_1) {
    const uint32_t *q = reinterpret_cast<const uint32_t *>(in) + px;
    if (y - 2 >= 0 && y - 2 < H) p.v[0].x = __ldg(q - 2 * (int64_t)W);
    if (y - 1 >= 0 && y - 1 < H) p.v[0].y = __ldg(q - (int64_t)W);
    if (y < H) p.v[0].z = __ldg(q);
    if (y + 1 < H) p.v[0].w = __ldg(q + W);
    if (y + 2 < H) p.v[1].x = __ldg(q + 2 * (int64_t)W);
  } else if (y >= 0 && y < H) {
#pragma unroll
    for (int k = 0; k < RcPx<IN>::NV; k++) p.v[k] = __ldg(reinterpret_cast<const uint4 *>(in) + px * RcPx<IN>::NV + k);
  }
}
// into slot position d of an input row (planes RC_PLANE apart)
template <int IN>
__device__ __forceinline__ void rc_store_px(const RcPx<IN> &p, uint8_t *d) {
  if constexpr (IN == RC_F32_1) {
    // K = 3 ky + part, and a zero
    uint32_t h[5], m[5], l[5];
    split3_bf16(__uint_as_float(p.v[0].x), h[0], m[0], l[0]);
    split3_bf16(__uint_as_float(p.v[0].y), h[1], m[1], l[1]);
    split3_bf16(__uint_as_float(p.v[0].z), h[2], m[2], l[2]);
    split3_bf16(__uint_as_float(p.v[0].w), h[3], m[3], l[3]);
    split3_bf16(__uint_as_float(p.v[1].x), h[4], m[4], l[4]);
    *reinterpret_cast<uint4 *>(d) =
        make_uint4(pack_hi(h[0], m[0]), pack_hi(l[0], h[1]), pack_hi(m[1], l[1]), pack_hi(h[2], m[2]));
    *reinterpret_cast<uint4 *>(d + RC_PLANE) =
        make_uint4(pack_hi(l[2], h[3]), pack_hi(m[3], l[3]), pack_hi(h[4], m[4]), l[4] >> 16);
  } else {
#pragma unroll
    for (int half = 0; half < 2; half++) {
      uint32_t h[8], m[8], l[8];
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const uint4 u = p.v[2 * half + k];
        split3_bf16(__uint_as_float(u.x), h[4 * k], m[4 * k], l[4 * k]);
        split3_bf16(__uint_as_float(u.y), h[4 * k + 1], m[4 * k + 1], l[4 * k + 1]);
        split3_bf16(__uint_as_float(u.z), h[4 * k + 2], m[4 * k + 2], l[4 * k + 2]);
        split3_bf16(__uint_as_float(u.w), h[4 * k + 3], m[4 * k + 3], l[4 * k + 3]);
      }
      *reinterpret_cast<uint4 *>(d + half * RC_PLANE) =
          make_uint4(pack_hi(h[0], h[1]), pack_hi(h[2], h[3]), pack_hi(h[4], h[5]), pack_hi(h[6], h[7]));
      *reinterpret_cast<uint4 *>(d + (2 + half) * RC_PLANE) =
          make_uint4(pack_hi(m[0], m[1]), pack_hi(m[2], m[3]), pack_hi(m[4], m[5]), pack_hi(m[6], m[7]));
      *reinterpret_cast<uint4 *>(d + (4 + half) * RC_PLANE) =
          make_uint4(pack_hi(l[0], l[1]), pack_hi(l[2], l[3]), pack_hi(l[4], l[5]), pack_hi(l[6], l[7]));
    }
  }
}

// Element (ky, k, n) of the weight operand: k the layer's output channel (a
// one-channel gradient: k = 3 ky + part, the parts share a weight), column
// n = kx * 16 + the layer's input channel.
template <int IN>
__device__ __forceinline__ __nv_bfloat16 rc_weight(const __nv_bfloat16 *__restrict__ w, int ky, int k, int n) {
  if (IN == RC_F32_1 && k >= 15) return __float2bfloat16_rn(0.0f);
  const int kx = n >> 4, ci = n & 15, co = IN == RC_F32_1 ? 0 : k, y = IN == RC_F32_1 ? k / 3 : ky;
  return __ldg(w + (co * CNN_HID + ci) * TAPS + (TAPS - 1 - (y * 5 + kx)));
}

template <int IN>
__global__ void __launch_bounds__(RC_THREADS, 1) k_grad_rows(const float *__restrict__ in, int W, int H, int n_img,
                                                            const __nv_bfloat16 *__restrict__ w,
                                                            float *__restrict__ out,
                                                            const __nv_bfloat16 *__restrict__ act) {
  using I = RcIn<IN>;
  constexpr int N = RC_N;
  extern __shared__ __align__(1024) uint8_t rsm[];
  uint8_t *ring = rsm;
  uint8_t *wsm = rsm + RC_SLOTS * I::PAIR;  // [ky][k half][n][8] bf16
  uint64_t *full = reinterpret_cast<uint64_t *>(wsm + I::KY * 2 * N * 16);
  uint64_t *empty = full + RC_SLOTS, *dfull = empty + RC_SLOTS, *dempty = dfull + RC_MMA_WARPS,
           *drain = dempty + RC_MMA_WARPS;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile uint32_t *stop = tmem_slot + 1;
  static_assert((2 * RC_SLOTS + 2 * RC_MMA_WARPS + 2) * 8 <= 512, "barrier words");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool loader = warp >= RC_EPI_WARPS && warp < RC_EPI_WARPS + RC_LOAD_WARPS;
  const int pairs = (H + 1) / 2, strips = (W + RC_OUT - 1) / RC_OUT;
  const int64_t total = (int64_t)strips * n_img * pairs;
  RcSeg seg;
  seg.r = total * blockIdx.x / gridDim.x;
  seg.end = total * (blockIdx.x + 1) / gridDim.x;

  // Loaders: one pixel of each of a pair's two input rows per thread (pair g of
  // the block's sequence goes to ring slot g % RC_SLOTS), RC_AHEAD pairs in
  // flight, the first of them while the block is set up.
  const int slot = tid - 32 * RC_EPI_WARPS;
  const int dx = (slot >> 5) * 28 + lane - 2;
  RcSeg c = seg;
  int ci = 0;  // the segment's next input pair to fetch, 0 .. len + HALO - 1
  RcPx<IN> p[RC_AHEAD][2];
  auto fetch = [&](RcPx<IN> (&q)[2]) {
    if (c.r >= c.end) return;
    const int gx = c.x0 + dx, gy = c.y0 - I::HALO + 2 * ci;
    const bool in_x = gx >= 0 && gx < W;
    const size_t px = ((size_t)c.img * H + gy) * W + gx;
    rc_load_px<IN>(q[0], in, in_x, gy, H, W, px);
    rc_load_px<IN>(q[1], in, in_x, gy + 1, H, W, px + W);
    if (++ci < c.len + I::HALO) return;
    c.r += c.len;
    ci = 0;
    if (c.r < c.end) rc_seg(c, pairs, strips);
  };
  if (loader) {
    if (c.r < c.end) rc_seg(c, pairs, strips);
#pragma unroll
    for (int k = 0; k < RC_AHEAD; k++) fetch(p[k]);
  } else {
    // (all of a thread's weights in flight at once)
    constexpr int SETUP = RC_THREADS - 32 * RC_LOAD_WARPS, WN = I::KY * 16 * N,
                  PER = (WN + SETUP - 1) / SETUP;
    const int t = warp < RC_EPI_WARPS ? tid : tid - 32 * RC_LOAD_WARPS;
    __nv_bfloat16 v[PER];
#pragma unroll
    for (int k = 0; k < PER; k++) {
      const int i = t + k * SETUP, n = (i >> 3) % N, r = (i >> 3) / N;
      if (i < WN) v[k] = rc_weight<IN>(w, r >> 1, (r & 1) * 8 + (i & 7), n);
    }
#pragma unroll
    for (int k = 0; k < PER; k++)
      if (t + k * SETUP < WN) reinterpret_cast<__nv_bfloat16 *>(wsm)[t + k * SETUP] = v[k];
    if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                   "r"(RC_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 32) {
      auto init = [](uint64_t *b, uint32_t n) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(n));
      };
      for (int k = 0; k < RC_SLOTS; k++) init(full + k, RC_LOAD_WARPS), init(empty + k, RC_MMA_WARPS);
      for (int k = 0; k < RC_MMA_WARPS; k++) init(dfull + k, 1), init(dempty + k, RC_EPI_WARPS / 2);
      init(drain, RC_MMA_WARPS);
      *stop = 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (loader) {
    // input pairs of the whole share: its output pairs, and the halo of each segment
    const int64_t segs = seg.r < seg.end ? (seg.end - 1) / pairs - seg.r / pairs + 1 : 0;
    const uint32_t count = (uint32_t)(seg.end - seg.r + I::HALO * segs);
    // (a pair's registers are filled again in place: moving one that a load
    // still owes would wait for that load)
    bool ok = true;
    uint8_t *const dst = ring + slot * 16;
    uint32_t sl = 0, par = 1;  // ring slot; parity of the wait for it (at once in the first turn)
    for (uint32_t g0 = 0; g0 < count && ok; g0 += RC_AHEAD) {
#pragma unroll
      for (int k = 0; k < RC_AHEAD; k++) {
        if (g0 + (uint32_t)k >= count) break;
        ok = __all_sync(0xffffffffu, tc_wait(empty + sl, par, stop));  // (the warp stops as one: its lanes meet below)
        if (!ok) break;
        rc_store_px<IN>(p[k][0], dst + sl * I::PAIR);
        rc_store_px<IN>(p[k][1], dst + sl * I::PAIR + I::ROW);
        __syncwarp();
        if (lane == 0) tc_arrive(full + sl);
        if (++sl == RC_SLOTS) sl = 0, par ^= 1;
        fetch(p[k]);
      }
    }
  } else if (warp >= RC_EPI_WARPS) {
    if (lane == 0) {
      // MMAs: of every segment, issuer m takes output rows m, m + 4, ... into its
      // own accumulator m (four chains of MMAs run side by side: those of one
      // accumulator wait for one another).  Its row of output pair k reads input
      // pairs k .. k + HALO, there when the last one is (the loaders take
      // them in order).  Every issuer releases every input pair once, in order:
      // by a commit after its last row that reads it, or, reading none of it,
      // after it has passed; so no phase of a slot is missed.
      const uint32_t m = (uint32_t)(warp - RC_EPI_WARPS - RC_LOAD_WARPS);
      const uint32_t rbase = smem_addr(ring), wbase = smem_addr(wsm);
      uint32_t g = 0, dpar = 1;  // the segment's first input pair; parity of the wait for the accumulator
      bool ok = true;
      auto wait_full = [&](uint32_t gi) { return tc_wait(full + gi % RC_SLOTS, (gi / RC_SLOTS) & 1, stop); };
      while (seg.r < seg.end && ok) {
        rc_seg(seg, pairs, strips);
        const uint32_t len = (uint32_t)seg.len;
        uint32_t p = 0;  // the segment's next input pair to release
        for (uint32_t k = m >> 1;; k += 2) {
          const uint32_t upto = k < len ? k : len + I::HALO;
          for (; p < upto && ok; p++) {
            ok = wait_full(g + p);
            if (ok) tc_arrive(empty + (g + p) % RC_SLOTS);
          }
          if (k >= len || !ok) break;
          const uint32_t gi = g + k;
          const uint32_t r0 = rbase + gi % RC_SLOTS * I::PAIR, r1 = rbase + (gi + 1) % RC_SLOTS * I::PAIR,
                         r2 = rbase + (gi + 2) % RC_SLOTS * I::PAIR;
          // (without a halo the output row's operand is the one ring row r0)
          const uint32_t rb[5] = {m & 1 ? r0 + I::ROW : r0, m & 1 ? r1 : r0 + I::ROW, m & 1 ? r1 + I::ROW : r1,
                                  m & 1 ? r2 : r1 + I::ROW, m & 1 ? r2 + I::ROW : r2};
          ok = wait_full(gi + I::HALO) && tc_wait(dempty + m, dpar, stop);
          if (!ok) break;
          dpar ^= 1;
          // the loaders' stores, acquired through their barrier, ordered
          // before the tensor core's reads
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          // (the lowest parts first: the accumulator rounds each sum toward
          // zero, and the small parts' sums lose least while they are alone)
#pragma unroll
          for (int part = I::PARTS - 1; part >= 0; part--)
#pragma unroll
            for (int ky = 0; ky < I::KY; ky++)
              tc_mma(tmem + m * N, tc_desc(rb[ky] + part * 2 * RC_PLANE, RC_PLANE, 128),
                     tc_desc(wbase + (uint32_t)(ky * 2 * N * 16), N * 16, 128), tc_idesc(N),
                     (ky || part < I::PARTS - 1) ? 1u : 0u);
          tc_commit(dfull + m);
          // the input pairs this issuer's next row does not read
          const uint32_t last = (k + 2 < len && I::HALO > 1) ? k + 1 : k + I::HALO;
          for (; p <= last; p++) tc_commit(empty + (g + p) % RC_SLOTS);
        }
        g += len + I::HALO;
        seg.r += seg.len;
      }
      // every MMA and commit done before the block's memory is given back
      tc_commit(drain);
      uint32_t never = 0u;
      tc_wait(drain, 0, &never);
    }
  } else {
    // Epilogue: a group of four warps for each row of a pair; it takes
    // accumulators row and row + 2 in turn, from row in every segment
    const int quad = warp & 3, row = warp >> 2;
    const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16);
    uint32_t par = 0;  // bit d: parity of the next wait for accumulator d
    while (seg.r < seg.end) {
      rc_seg(seg, pairs, strips);
      uint32_t d = (uint32_t)row;
      const int gx = seg.x0 + quad * 28 + lane;
      for (int i = 0; i < seg.len; i++) {
        const int gy = seg.y0 + 2 * i + row;
        const size_t px = ((size_t)seg.img * H + gy) * W + gx;
        const bool inside = lane < 28 && gx < W && gy < H;
        uint4 am[2];
        if (inside) {
          am[0] = __ldg(reinterpret_cast<const uint4 *>(act + px * 16));
          am[1] = __ldg(reinterpret_cast<const uint4 *>(act + px * 16) + 1);
        }
        const bool ok = tc_wait(dfull + d, (par >> d) & 1, stop);
        __syncwarp();  // (the reads of tensor memory are by whole warps)
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t v[N / 16][16];
#pragma unroll
        for (int kx = 0; kx < N / 16; kx++) tmem_ld16(trow + d * N + kx * 16, v[kx]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (lane == 0) tc_arrive(dempty + d);
        par ^= 1u << d;
        d ^= 2;
        float a[16];
#pragma unroll
        for (int k = 0; k < 16; k++) {
          a[k] = __uint_as_float(v[0][k]);
#pragma unroll
          for (int kx = 1; kx < 5; kx++) a[k] += __shfl_down_sync(0xffffffffu, __uint_as_float(v[kx][k]), kx);
          if (!ok) a[k] = __uint_as_float(0x7FC00000u);  // NaN: the accumulators were not read
        }
        if (inside) {
          const __nv_bfloat16 *ab = reinterpret_cast<const __nv_bfloat16 *>(am);
          float4 *dst = reinterpret_cast<float4 *>(out + px * 16);
#pragma unroll
          for (int k = 0; k < 16; k += 4) {
            float4 o;
            o.x = __bfloat162float(ab[k]) > 0.0f ? a[k] : 0.0f;
            o.y = __bfloat162float(ab[k + 1]) > 0.0f ? a[k + 1] : 0.0f;
            o.z = __bfloat162float(ab[k + 2]) > 0.0f ? a[k + 2] : 0.0f;
            o.w = __bfloat162float(ab[k + 3]) > 0.0f ? a[k + 3] : 0.0f;
            dst[k / 4] = o;
          }
        }
        __syncwarp();
      }
      seg.r += seg.len;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(RC_COLS));
}

// ------------------------------------------- tensor-core weight gradients
//
// dW[co][ci][ky][kx] = sum over pixels p of dy[p][co] * x[p + (ky-2, kx-2)][ci],
// db[co] = sum of dy[co]: a GEMM whose contraction runs over the pixels, on
// the 5th-generation tensor cores.  Both operands lie in shared memory pixel
// after pixel with 8 channels (16 bytes) each, which is the M- and N-major
// unswizzled canonical layout (core matrices of 8 pixels x 8 channels, 128
// bytes; the next 8 pixels of K at LBO = 128, the next 8 channels at SBO).
//   A (M = 128): 16 groups of 8 channels of x, the group stride running over
//     (row, plane) of the tile, so one MMA holds 8 rows of 16 channels;
//   B (N = G * NS): G rows of dy.  dy is FP32 and enters as three BF16 parts
//     (top, middle and low 8 bits of the significand, by truncation), whose
//     sum is dy exactly: with x in BF16 every product is exact, as in FP32;
//   D[row j of x][row i of dy] is the gradient for ky = j - i; the shift kx is
//     the start address of A's descriptor, one accumulator per kx.
// The accumulators are emptied into FP32 registers after every tile (16 or
// 8 MMAs each), so no long sum runs in the tensor core's accumulator.
// Layer 1 has one plane of 8 channels: its second plane is the same pixels
// one to the right, so that one accumulator serves two kx.
//
// What bounds it: shared-memory operand reads, (128 + N) x 32 bytes per MMA
// (56 of 128-byte reads against 48 cycles of math at N = 96), so G = 2 rows of dy
// per MMA for the 16-channel dy (5 x 96 columns of the 512 of tensor memory;
// one row needs 220 operand-read cycles per 16 pixels, two 140) and 4 rows
// for layer 3's single channel.  Measured on four 640x480 images: layers 2, 1 and 3 take 85,
// 66 and 42 us (an MMA about 90 cycles, the flush of the accumulators a tenth),
// with one (co, ci) pair per thread on the CUDA cores, 26 shared-memory reads
// per 25 FMAs, 969, 371 and 472 us.  Errors against 64 bits (relative L2 of the
// whole gradient): 2.2e-7 against 8.7e-7.
enum WgKind { WG_L1 = 1, WG_L2 = 2, WG_L3 = 3 };
constexpr int WG_THREADS = 256;
constexpr int WG_W = 64, WG_R = 8;     // dy pixels of a tile
constexpr int WG_XPX = 72;             // x pixels of a tile row: 64 + 4, whole 128-byte core matrices
constexpr int WG_XROWS = WG_R + 6;     // 12 rows of x; the last MMA's unused groups reach two further
constexpr int WG_XROW_BYTES = 2 * WG_XPX * 16;
constexpr int WG_XBYTES = WG_XROWS * WG_XROW_BYTES;

template <int KIND>
struct WgTraits {
  static constexpr int CO = KIND == WG_L3 ? 1 : 16;           // channels of dy
  static constexpr int CI = KIND == WG_L1 ? CNN_IN : CNN_HID;  // channels of x
  static constexpr int G = KIND == WG_L3 ? 4 : 2;              // rows of dy per MMA
  static constexpr int NS = KIND == WG_L3 ? 8 : 48;            // columns of a dy row: its channels' three parts
  static constexpr int N = G * NS;
  static constexpr int NKX = KIND == WG_L1 ? 3 : 5;            // accumulators
  static constexpr int KX_STEP = KIND == WG_L1 ? 2 : 1;
  static constexpr int COLS = KIND == WG_L3 ? 256 : 512;       // tensor-memory columns allocated
  static constexpr int GBYTES = WG_R * (NS / 8) * WG_W * 16;   // dy parts of a tile
  static constexpr int BUF = WG_XBYTES + GBYTES;
  static constexpr int DW = CO * CI * TAPS;
  static constexpr int ACC = KIND == WG_L3 ? 2 : 16;           // accumulators per kx and thread
  static_assert(NKX * N <= COLS, "accumulators fit the allocation");
  static_assert(DW * 4 + 64 * 4 <= BUF, "the block's sums reuse a tile buffer");
};
// (the blocks that allocate all 512 columns leave no room for a second one)
template <int KIND>
constexpr size_t wg_smem_bytes() {
  return 2 * (size_t)WgTraits<KIND>::BUF + 64;
}
static_assert((WG_XPX * 16) % 128 == 0 && WG_XBYTES % 128 == 0 && WgTraits<WG_L2>::BUF % 128 == 0 &&
                  WgTraits<WG_L3>::BUF % 128 == 0,
              "tile copies land on 128-byte boundaries");
static_assert(wg_smem_bytes<WG_L1>() > 114 * 1024 && wg_smem_bytes<WG_L2>() > 114 * 1024, "one block per SM");

// M = 128, D FP32, A and B BF16, both M/N-major
template <int N>
__host__ __device__ constexpr uint32_t wg_idesc() {
  return tc_idesc(N) | (1u << 15) | (1u << 16);
}

template <int KIND>
__global__ void __launch_bounds__(WG_THREADS) k_wgrad_tc(const __grid_constant__ CUtensorMap tile,
                                                         const float *__restrict__ dy, int W, int H, int n_img,
                                                         float *__restrict__ dw, float *__restrict__ db) {
  using T = WgTraits<KIND>;
  extern __shared__ __align__(1024) uint8_t wsm[];
  uint64_t *mbar = reinterpret_cast<uint64_t *>(wsm + 2 * T::BUF);  // [0], [1]: x of a buffer; [2]: MMAs
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(mbar + 3);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)),
                 "r"(T::COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int k = 0; k < 3; k++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar + k)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const int tiles_x = (W + WG_W - 1) / WG_W, tiles_y = (H + WG_R - 1) / WG_R;
  const int total = tiles_x * tiles_y * n_img;
  struct Pos {
    int img, x0, y0;
  };
  auto pos_of = [&](int t) {
    Pos p;
    p.img = t / (tiles_x * tiles_y);
    const int rest = t % (tiles_x * tiles_y);
    p.x0 = (rest % tiles_x) * WG_W;
    p.y0 = (rest / tiles_x) * WG_R;
    return p;
  };
  // x of a tile: (8 + 4) rows of two planes, each row of a plane one copy
  // (zero outside the image), issued by the first 24 lanes of warp 1
  auto load_x = [&](const Pos &p, int b) {
    if (warp != 1) return;
    const uint32_t bar = smem_addr(mbar + b), dst = smem_addr(wsm + b * T::BUF);
    if (lane == 0)
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                   "r"((uint32_t)((WG_R + 4) * WG_XROW_BYTES))
                   : "memory");
    __syncwarp();
    if (lane < 2 * (WG_R + 4)) {
      const int r = lane >> 1, pl = lane & 1;
      const uint32_t d = dst + (uint32_t)(r * WG_XROW_BYTES + pl * WG_XPX * 16);
      if constexpr (KIND == WG_L1)
        tma_load_4d(d, &tile, 0, p.x0 - 2 + pl, p.y0 - 2 + r, p.img, bar);
      else
        tma_load_5d(d, &tile, 0, pl, p.x0 - 2, p.y0 - 2 + r, p.img, bar);
    }
    __syncwarp();
  };
  // dy of a tile, split: [row][part, channel plane][pixel][8 channels]; zero
  // outside the image.  The running sums of what a thread reads are its share
  // of the bias gradient.
  float bias[KIND == WG_L3 ? 1 : 4] = {};
  auto load_g = [&](const Pos &p, int b) {
    uint8_t *gs = wsm + b * T::BUF + WG_XBYTES;
    const size_t base = (size_t)p.img * H * W;
    if constexpr (KIND == WG_L3) {
#pragma unroll
      for (int it = 0; it < WG_W * WG_R / WG_THREADS; it++) {
        const int i = it * WG_THREADS + tid;
        const int gx = p.x0 + i % WG_W, gy = p.y0 + i / WG_W;
        const float v = (gx < W && gy < H) ? __ldg(dy + base + (size_t)gy * W + gx) : 0.0f;
        bias[0] += v;
        uint32_t h, m, l;
        split3_bf16(v, h, m, l);
        *reinterpret_cast<uint4 *>(gs + (size_t)i * 16) = make_uint4(pack_hi(h, m), l >> 16, 0u, 0u);
      }
    } else {
      const int q = tid & 3;  // this thread's four channels
      float4 f[8];
#pragma unroll
      for (int it = 0; it < 8; it++) {
        const int px = it * (WG_THREADS / 4) + (tid >> 2);
        const int gx = p.x0 + px % WG_W, gy = p.y0 + px / WG_W;
        f[it] = (gx < W && gy < H)
                    ? __ldg(reinterpret_cast<const float4 *>(dy + (base + (size_t)gy * W + gx) * 16) + q)
                    : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
#pragma unroll
      for (int it = 0; it < 8; it++) {
        const int px = it * (WG_THREADS / 4) + (tid >> 2);
        const float v[4] = {f[it].x, f[it].y, f[it].z, f[it].w};
        uint32_t h[4], m[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          bias[k] += v[k];
          split3_bf16(v[k], h[k], m[k], l[k]);
        }
        uint8_t *d = gs + (size_t)(px / WG_W) * (6 * WG_W * 16) + (size_t)(q >> 1) * (WG_W * 16) +
                     (size_t)(px % WG_W) * 16 + (q & 1) * 8;
        *reinterpret_cast<uint2 *>(d) = make_uint2(pack_hi(h[0], h[1]), pack_hi(h[2], h[3]));
        *reinterpret_cast<uint2 *>(d + 2 * WG_W * 16) = make_uint2(pack_hi(m[0], m[1]), pack_hi(m[2], m[3]));
        *reinterpret_cast<uint2 *>(d + 4 * WG_W * 16) = make_uint2(pack_hi(l[0], l[1]), pack_hi(l[2], l[3]));
      }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  };
  // the tile's MMAs, by one thread once x has landed; returns whether it has
  auto issue = [&](int b, uint32_t parity) -> uint32_t {
    const uint32_t ok = mbar_wait(smem_addr(mbar + b), parity);
    if (!ok) return 0u;
    const uint32_t xb = smem_addr(wsm + b * T::BUF), gb = xb + WG_XBYTES;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    for (int ip = 0; ip < WG_R / T::G; ip++)
      for (int ch = 0; ch < WG_W / 16; ch++) {
        const uint64_t bd = tc_desc(gb + (uint32_t)(ip * T::G * (T::NS / 8) * WG_W * 16 + ch * 256), 128, WG_W * 16);
#pragma unroll
        for (int k = 0; k < T::NKX; k++) {
          const uint64_t ad = tc_desc(
              xb + (uint32_t)(ip * T::G * WG_XROW_BYTES + (ch * 16 + k * T::KX_STEP) * 16), 128, WG_XPX * 16);
          tc_mma(tmem + (uint32_t)(k * T::N), ad, bd, wg_idesc<T::N>(), (ip | ch) ? 1u : 0u);
        }
      }
    tc_commit(mbar + 2);
    return 1u;
  };
  const int quad = warp & 3, half = warp >> 2;
  const uint32_t trow = tmem + ((uint32_t)(32 * quad) << 16);
  float acc[T::NKX][T::ACC];
#pragma unroll
  for (int k = 0; k < T::NKX; k++)
#pragma unroll
    for (int c = 0; c < T::ACC; c++) acc[k][c] = 0.0f;
  int t = blockIdx.x;  // (below total: the grid has at most that many blocks)
  {
    const Pos first = pos_of(t);
    load_x(first, 0);
    load_g(first, 0);
  }
  __syncthreads();
  uint32_t pending_x = 0;  // (bit b: a copy into buffer b whose arrival nobody has waited for)
  int it = 0;
  bool bad = false;
  for (; t < total; t += gridDim.x, it++) {
    const int b = it & 1;
    bool ok = tid != 0 || issue(b, (uint32_t)((it >> 1) & 1));
    __syncwarp();
    // the next tile's operands while the MMAs run (their buffer's last
    // readers, the previous tile's MMAs, have finished)
    const int tn = t + (int)gridDim.x;
    pending_x = 0;
    if (tn < total) {
      const Pos nx = pos_of(tn);
      load_x(nx, b ^ 1);
      load_g(nx, b ^ 1);
      pending_x = 1u;
    }
    const uint32_t done = mbar_wait(smem_addr(mbar + 2), (uint32_t)(it & 1));
    ok = ok && done;
    const bool read = __all_sync(0xffffffffu, done != 0u);  // (the reads of tensor memory are by whole warps)
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (read) {
      if constexpr (KIND == WG_L3) {
#pragma unroll
        for (int k = 0; k < T::NKX; k++) {
          uint32_t v[16];  // rows 2 half, 2 half + 1 of dy
          tmem_ld16(trow + (uint32_t)(k * T::N + half * 16), v);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 2; i++)
            acc[k][i] += __uint_as_float(v[8 * i]) + (__uint_as_float(v[8 * i + 1]) + __uint_as_float(v[8 * i + 2]));
        }
      } else if (quad < 3) {  // (rows 6 and 7 of x meet neither row of dy)
#pragma unroll
        for (int k = 0; k < T::NKX; k++) {
          uint32_t h[16], m[16], l[16];  // row `half` of dy
          tmem_ld16(trow + (uint32_t)(k * T::N + half * T::NS), h);
          tmem_ld16(trow + (uint32_t)(k * T::N + half * T::NS + 16), m);
          tmem_ld16(trow + (uint32_t)(k * T::N + half * T::NS + 32), l);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int c = 0; c < 16; c++)
            acc[k][c] += __uint_as_float(h[c]) + (__uint_as_float(m[c]) + __uint_as_float(l[c]));
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    bad = __syncthreads_or(ok ? 0 : 1) != 0;
    if (bad) break;
  }
  // A wait that gave up may leave copies or MMAs in flight: wait for them once
  // more (bounded again) before their memory is given back; the gradients
  // become NaN.
  if (bad) {
    mbar_wait(smem_addr(mbar + 2), (uint32_t)(it & 1));
    mbar_wait(smem_addr(mbar + (it & 1)), (uint32_t)((it >> 1) & 1));
    if (pending_x) mbar_wait(smem_addr(mbar + ((it & 1) ^ 1)), (uint32_t)(((it + 1) >> 1) & 1));
    __syncthreads();
  }
  // the block's gradients in shared memory: row i of dy meets row j of x at
  // ky = j - i, so each element is met once per i, in G steps
  float *s_dw = reinterpret_cast<float *>(wsm);
  float *s_db = s_dw + T::DW;
  for (int i = tid; i < T::DW + T::CO; i += WG_THREADS) s_dw[i] = 0.0f;
  __syncthreads();
  const int m = 32 * quad + lane, j = m >> 4, pl = (m >> 3) & 1, c8 = m & 7;
  const int ci = KIND == WG_L1 ? c8 : pl * 8 + c8;
#pragma unroll
  for (int i = 0; i < T::G; i++) {
    const int ky = j - i;
    const bool mine = KIND == WG_L3 ? (i >> 1) == half : i == half;
    if (mine && ky >= 0 && ky < 5 && ci < T::CI) {
#pragma unroll
      for (int k = 0; k < T::NKX; k++) {
        const int kx = k * T::KX_STEP + (KIND == WG_L1 ? pl : 0);
        if (kx < 5) {
          if constexpr (KIND == WG_L3) {
            s_dw[ci * TAPS + ky * 5 + kx] += acc[k][i & 1];
          } else {
#pragma unroll
            for (int co = 0; co < 16; co++) s_dw[(co * T::CI + ci) * TAPS + ky * 5 + kx] += acc[k][co];
          }
        }
      }
    }
    __syncthreads();
  }
  // the bias: lanes of the same channels, then one add per warp
  if constexpr (KIND == WG_L3) {
    float v = bias[0];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) atomicAdd(s_db, v);
  } else {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      float v = bias[k];
#pragma unroll
      for (int o = 16; o > 2; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane < 4) atomicAdd(s_db + 4 * lane + k, v);
    }
  }
  __syncthreads();
  for (int i = tid; i < T::DW; i += WG_THREADS) atomicAdd(dw + i, bad ? __int_as_float(0x7FC00000) : s_dw[i]);
  for (int i = tid; i < T::CO; i += WG_THREADS) atomicAdd(db + i, bad ? __int_as_float(0x7FC00000) : s_db[i]);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(T::COLS));
}

// Network input per pixel: depth z (m), the unit normal from central
// differences of the back-projected neighbours (zero unless all four are
// valid), and the validity flag.
__global__ void k_cnn_features(const __grid_constant__ FeatureImages images, int W, int H, float scaling,
                               __nv_bfloat16 *__restrict__ feat) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, img = blockIdx.z;
  if (x >= W) return;
  const uint16_t *__restrict__ d = images.depth[img];
  const float fx = images.K[img][0], fy = images.K[img][1], cx = images.K[img][2], cy = images.K[img][3];
  auto zat = [&](int xx, int yy) -> float {
    return (xx < 0 || yy < 0 || xx >= W || yy >= H) ? 0.0f : scaling * (float)__ldg(d + (size_t)yy * W + xx);
  };
  const float z = zat(x, y);
  const float zl = zat(x - 1, y), zr = zat(x + 1, y), zu = zat(x, y - 1), zd = zat(x, y + 1);
  float nx = 0.0f, ny = 0.0f, nz = 0.0f;
  if (z > 0.0f && zl > 0.0f && zr > 0.0f && zu > 0.0f && zd > 0.0f) {
    // a = P(x+1) - P(x-1), b = P(y+1) - P(y-1); n = b x a faces the camera
    const float ax = ((float)(x + 1) - cx) * zr / fx - ((float)(x - 1) - cx) * zl / fx;
    const float ay = ((float)y - cy) * (zr - zl) / fy;
    const float az = zr - zl;
    const float bx = ((float)x - cx) * (zd - zu) / fx;
    const float by = ((float)(y + 1) - cy) * zd / fy - ((float)(y - 1) - cy) * zu / fy;
    const float bz = zd - zu;
    nx = by * az - bz * ay;
    ny = bz * ax - bx * az;
    nz = bx * ay - by * ax;
    const float len = sqrtf(nx * nx + ny * ny + nz * nz);
    if (len > 0.0f) {
      nx /= len;
      ny /= len;
      nz /= len;
    } else {
      nx = ny = nz = 0.0f;
    }
  }
  uint4 u;
  __nv_bfloat16 *b = reinterpret_cast<__nv_bfloat16 *>(&u);
  b[0] = __float2bfloat16_rn(z);
  b[1] = __float2bfloat16_rn(nx);
  b[2] = __float2bfloat16_rn(ny);
  b[3] = __float2bfloat16_rn(nz);
  b[4] = __float2bfloat16_rn(z > 0.0f ? 1.0f : 0.0f);
  b[5] = b[6] = b[7] = __float2bfloat16_rn(0.0f);
  reinterpret_cast<uint4 *>(feat)[((size_t)img * H + y) * W + x] = u;
}

// Mean squared error over labelled pixels (target >= 0; negative = no
// label): dpred = 2 (pred - target) * inv_count, loss += sum * inv_count.
__global__ void k_cnn_mse(const float *__restrict__ pred, const float *__restrict__ target, int64_t n,
                          float inv_count, float *__restrict__ dpred, double *__restrict__ loss) {
  double local = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float y = target[i];
    float g = 0.0f;
    if (y >= 0.0f) {
      const float e = pred[i] - y;
      g = 2.0f * e * inv_count;
      local += (double)e * (double)e;
    }
    dpred[i] = g;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0 && local != 0.0) atomicAdd(loss, local * (double)inv_count);
}

// Adam on the FP32 master weights; the BF16 copy the kernels use is written
// from the updated master, and the gradient is cleared for the next step.
__global__ void k_cnn_adam(float *__restrict__ master, __nv_bfloat16 *__restrict__ params, float *__restrict__ grad,
                           float *__restrict__ m, float *__restrict__ v, int n, float lr, float b1, float b2,
                           float eps, float bc1, float bc2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = grad[i];
  const float mi = b1 * m[i] + (1.0f - b1) * g;
  const float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float w = master[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  master[i] = w;
  params[i] = __float2bfloat16_rn(w);
  grad[i] = 0.0f;
}

// ------------------------------------------------------------------ raycast

constexpr int RAYCAST_MAX_STEPS = 4096;

// The octree slot at the end of a voxel's descent: every voxel of its box has
// the same finest leaf (UINT32_MAX: none).
struct RaySlot {
  uint32_t x, y, z, edge;  // (edge 0: no voxel)
  uint32_t leaf;
};
__device__ __forceinline__ bool in_slot(const RaySlot &S, uint32_t x, uint32_t y, uint32_t z) {
  return x - S.x < S.edge && y - S.y < S.edge && z - S.z < S.edge;
}
__device__ __forceinline__ RaySlot ray_slot(const uint32_t *__restrict__ tree, uint32_t n, uint32_t leaves_max,
                                            uint32_t x, uint32_t y, uint32_t z) {
  RaySlot S{0, 0, 0, 0, UINT32_MAX};
  uint32_t half = n >> 1, branch = 0;
  for (int level = 0; level < 16 && half >= (uint32_t)BL; level++) {
    const uint32_t co = (x >= S.x + half) * 1u + (y >= S.y + half) * 2u + (z >= S.z + half) * 4u;
    const uint32_t leaf = __ldg(tree + branch + co);
    if (leaf < leaves_max) S.leaf = leaf;
    const uint32_t child = __ldg(tree + branch + co + 8);
    S.x += half * ((co & 1) != 0);
    S.y += half * ((co & 2) != 0);
    S.z += half * ((co & 4) != 0);
    S.edge = half;
    if (child >= PENDING) break;  // BRANCHINIT (no child)
    branch = child;
    half >>= 1;
  }
  return S;
}

// Depth (m) of the first surface crossing of pixel (x, y)'s ray within
// +-window of its measured depth: the fused SDF of the finest brick
// (trilinear where the 8 surrounding voxels lie in the brick and are
// weighted, else the nearest voxel) sampled every `step` metres of depth,
// a change from negative (in front of the surface) to non-negative, both
// samples weighted, linearly interpolated -- or, entering a weighted band
// from unallocated space with 0 <= s < the truncation distance, t - s.
// 0 where the pixel has no depth, -1 where no surface lies in the window.
//
// What bounds it: the latency of dependent loads, sample after sample: a descent
// of the octree (eight levels) and 16 voxel loads each.  Samples half a voxel
// apart mostly stay in the octree slot and the voxel cube of the sample before,
// so a thread keeps both, with the cube's values; a warp takes 8x4 pixels, whose
// rays share bricks.  640x480, 0.15 m either side in steps of 2.5 mm: 473 -> 293 us.
constexpr int RAY_THREADS = 128, RAY_W = 16, RAY_H = 8;  // pixels of a block: warps of 8x4, two by two
__global__ void __launch_bounds__(RAY_THREADS) k_raycast(RaycastMap m, CamF p, int W, int H,
                                                        const uint16_t *__restrict__ depth, float scaling,
                                                        float window, float step, float *__restrict__ out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = blockIdx.x * RAY_W + 8 * (warp & 1) + (lane & 7), y = blockIdx.y * RAY_H + 4 * (warp >> 1) + (lane >> 3);
  if (x >= W || y >= H) return;
  const float d0 = scaling * (float)__ldg(depth + (size_t)y * W + x);
  float res = 0.0f;
  if (d0 > 0.0f) {
    res = -1.0f;
    const float rx = ((float)x - p.cx) / p.fx, ry = ((float)y - p.cy) / p.fy;
    const float t0 = fmaxf(d0 - window, 0.05f), t1 = d0 + window;
    bool prev_ok = false;
    float prev_s = 0.0f, prev_t = 0.0f, band = 0.0f;
    RaySlot slot{0, 0, 0, 0, UINT32_MAX};
    // the slot's leaf: its origin and voxel size, the cube of 8 voxels last
    // read (its number in the brick, values, all weighted), the voxel last read
    float ox = 0.0f, oy = 0.0f, oz = 0.0f, ls = 1.0f;
    int cube = -1, voxel = -1;
    float cv[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f}, vv = 0.0f;
    bool cube_ok = false, voxel_ok = false;
    const int nsteps = min((int)((t1 - t0) / step) + 1, RAYCAST_MAX_STEPS);
    for (int k = 0; k < nsteps; k++) {
      const float t = t0 + (float)k * step;
      const float cxm = rx * t, cym = ry * t;
      const float gx = p.r[0] * cxm + p.r[1] * cym + p.r[2] * t + p.t[0];
      const float gy = p.r[3] * cxm + p.r[4] * cym + p.r[5] * t + p.t[1];
      const float gz = p.r[6] * cxm + p.r[7] * cym + p.r[8] * t + p.t[2];
      bool ok = false;
      float s = 0.0f;
      const int ix = __float2int_rn(gx), iy = __float2int_rn(gy), iz = __float2int_rn(gz);
      if (ix >= 0 && iy >= 0 && iz >= 0 && ix < (int)m.n && iy < (int)m.n && iz < (int)m.n) {
        if (!in_slot(slot, ix, iy, iz)) {
          const uint32_t before = slot.leaf;
          slot = ray_slot(m.tree, m.n, m.leaves_max, ix, iy, iz);
          if (slot.leaf != before) {
            cube = voxel = -1;
            if (slot.leaf != UINT32_MAX) {
              const ushort4 o = __ldg(m.leaf + slot.leaf);
              ox = (float)o.x, oy = (float)o.y, oz = (float)o.z, ls = (float)o.w;
              band = 0.99f * m.thr * ls;
            }
          }
        }
        if (slot.leaf != UINT32_MAX) {
          const float ux = (gx - ox) / ls, uy = (gy - oy) / ls, uz = (gz - oz) / ls;
          const int fx0 = (int)floorf(ux), fy0 = (int)floorf(uy), fz0 = (int)floorf(uz);
          const size_t base = (size_t)slot.leaf * 512;
          if (fx0 >= 0 && fy0 >= 0 && fz0 >= 0 && fx0 < 7 && fy0 < 7 && fz0 < 7) {
            // trilinear inside the brick when its 8 voxels are all weighted
            const int first = (fz0 * 8 + fy0) * 8 + fx0;
            if (first != cube) {
              cube = first;
              cube_ok = true;
#pragma unroll
              for (int c = 0; c < 8; c++) {
                const size_t vi = base + first + ((c >> 2) * 8 + ((c >> 1) & 1)) * 8 + (c & 1);
                const float w = m.fp16 ? __half2float(m.wgt16[vi]) : m.wgt[vi];
                cv[c] = m.fp16 ? __half2float(m.sdf16[vi]) : m.sdf[vi];
                cube_ok = cube_ok && w > 0.0f;
              }
            }
            if (cube_ok) {
              const float ax = ux - (float)fx0, ay = uy - (float)fy0, az = uz - (float)fz0;
              float acc = 0.0f;
#pragma unroll
              for (int c = 0; c < 8; c++) {
                const int dx = c & 1, dy = (c >> 1) & 1, dz = c >> 2;
                acc += (dx ? ax : 1.0f - ax) * (dy ? ay : 1.0f - ay) * (dz ? az : 1.0f - az) * cv[c];
              }
              s = acc;
              ok = true;
            }
          }
          if (!ok) {  // nearest voxel
            const int lx = min(max(__float2int_rn(ux), 0), 7);
            const int ly = min(max(__float2int_rn(uy), 0), 7);
            const int lz = min(max(__float2int_rn(uz), 0), 7);
            const int at = (lz * 8 + ly) * 8 + lx;
            if (at != voxel) {
              voxel = at;
              const float w = m.fp16 ? __half2float(m.wgt16[base + at]) : m.wgt[base + at];
              vv = m.fp16 ? __half2float(m.sdf16[base + at]) : m.sdf[base + at];
              voxel_ok = w > 0.0f;
            }
            if (voxel_ok) {
              s = vv;
              ok = true;
            }
          }
        }
      }
      if (ok && prev_ok && prev_s < 0.0f && s >= 0.0f) {
        res = prev_t + step * (-prev_s) / (s - prev_s);
        break;
      }
      // entering the band of a surface from unallocated space (its front
      // side lies in a brick no sample allocated): the along-ray SDF places
      // the surface at t - s
      if (ok && !prev_ok && k > 0 && s >= 0.0f && s < band) {
        res = t - s;
        break;
      }
      prev_ok = ok;
      prev_s = s;
      prev_t = t;
    }
  }
  out[(size_t)y * W + x] = res;
}

// ---------------------------------------------------------------- launchers

namespace {
std::mutex g_attr_mu;
unsigned long long g_attr_done = 0;  // devices whose kernels have their shared-memory limits set

template <int C, int COUT, int MODE>
cudaError_t set_conv_attr() {
  return cudaFuncSetAttribute(k_conv_quads<C, COUT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)cq_smem_bytes<C, COUT>());
}
template <int IN>
cudaError_t set_grad_attr() {
  return cudaFuncSetAttribute(k_grad_rows<IN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rc_smem_bytes<IN>());
}
template <int KIND>
cudaError_t set_wgrad_attr() {
  return cudaFuncSetAttribute(k_wgrad_tc<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)wg_smem_bytes<KIND>());
}

cudaError_t ensure_attrs() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(g_attr_mu);
  const unsigned long long bit = 1ull << (dev & 63);
  if (g_attr_done & bit) return cudaSuccess;
  cudaError_t r[] = {
      set_conv_attr<8, 16, CONV_RELU_BF16>(),
      set_conv_attr<16, 16, CONV_RELU_BF16>(),
      set_conv_attr<16, 1, CONV_F32>(),
      set_conv_attr<16, 1, CONV_CONF>(),
      set_grad_attr<RC_F32_1>(),
      set_grad_attr<RC_F32_16>(),
      set_wgrad_attr<WG_L1>(),
      set_wgrad_attr<WG_L2>(),
      set_wgrad_attr<WG_L3>(),
  };
  for (cudaError_t x : r)
    if (x != cudaSuccess) return x;
  g_attr_done |= bit;
  return cudaSuccess;
}

// Tensor-map encoder of the driver, looked up once (the library does not
// link the driver library itself).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// The copies of k_wgrad_tc over n images of W x H pixels, C = 8 or 16 BF16
// channels per pixel: WG_XPX pixels of a row of one 8-channel plane, zero
// outside the image (dimensions: 8 channels, [plane], x, y, image).
cudaError_t tile_map(CUtensorMap *m, const void *base, int C, int W, int H, int n) {
  const EncodeTiledFn f = encode_tiled();
  if (!f) return cudaErrorNotSupported;
  cuuint64_t dims[5], strides[4];
  cuuint32_t box[5], es[5] = {1, 1, 1, 1, 1};
  cuuint32_t rank;
  if (C == 16) {
    rank = 5;
    const cuuint64_t d[5] = {8, 2, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)n};
    const cuuint64_t st[4] = {16, 32, (cuuint64_t)W * 32, (cuuint64_t)W * H * 32};
    const cuuint32_t b[5] = {8, 1, WG_XPX, 1, 1};
    for (int i = 0; i < 5; i++) dims[i] = d[i], box[i] = b[i];
    for (int i = 0; i < 4; i++) strides[i] = st[i];
  } else {
    rank = 4;
    const cuuint64_t d[4] = {8, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)n};
    const cuuint64_t st[3] = {16, (cuuint64_t)W * 16, (cuuint64_t)W * H * 16};
    const cuuint32_t b[4] = {8, WG_XPX, 1, 1};
    for (int i = 0; i < 4; i++) dims[i] = d[i], box[i] = b[i];
    for (int i = 0; i < 3; i++) strides[i] = st[i];
  }
  const CUresult r = f(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(base), dims, strides, box, es,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int C, int COUT, int MODE>
void conv(const __nv_bfloat16 *in, int n, int W, int H, const __nv_bfloat16 *w, const __nv_bfloat16 *b, void *out,
          float inv_tau, uint32_t *err, int err_stride, cudaStream_t s) {
  const int64_t quads = (int64_t)((W + CQ_OUT - 1) / CQ_OUT) * n * ((H + 3) / 4);
  note_launch();
  k_conv_quads<C, COUT, MODE><<<(int)std::min<int64_t>(148, quads), CQ_THREADS, cq_smem_bytes<C, COUT>(), s>>>(
      in, W, H, n, w, b, out, inv_tau, err, err_stride);
}

template <int IN>
void input_grad(const float *g, int n, int W, int H, const __nv_bfloat16 *w, float *out, const __nv_bfloat16 *act,
                cudaStream_t s) {
  const int64_t pairs = (int64_t)((W + RC_OUT - 1) / RC_OUT) * n * ((H + 1) / 2);
  const int grid = (int)std::min<int64_t>(148, (pairs + RC_MIN_PAIRS - 1) / RC_MIN_PAIRS);
  note_launch();
  k_grad_rows<IN><<<grid, RC_THREADS, rc_smem_bytes<IN>(), s>>>(g, W, H, n, w, out, act);
}

template <int KIND>
cudaError_t wgrad(const __nv_bfloat16 *x, const float *dy, int n, int W, int H, float *dw, float *db, cudaStream_t s) {
  CUtensorMap m;
  const cudaError_t e = tile_map(&m, x, KIND == WG_L1 ? CNN_IN_STRIDE : CNN_HID, W, H, n);
  if (e != cudaSuccess) return e;
  const int tiles = ((W + WG_W - 1) / WG_W) * ((H + WG_R - 1) / WG_R) * n;
  note_launch();
  k_wgrad_tc<KIND><<<std::min(tiles, 148), WG_THREADS, wg_smem_bytes<KIND>(), s>>>(m, dy, W, H, n, dw, db);
  return cudaGetLastError();
}
}  // namespace

cudaError_t cnn_features_of(const FeatureImages &images, int n, int W, int H, float scaling, __nv_bfloat16 *feat,
                            cudaStream_t s) {
  if (n < 1 || n > FEATURE_IMAGES_MAX) return cudaErrorInvalidValue;
  note_launch();
  k_cnn_features<<<dim3((W + 127) / 128, H, n), 128, 0, s>>>(images, W, H, scaling, feat);
  return cudaGetLastError();
}

cudaError_t cnn_features(const uint16_t *depth, int n, int W, int H, float scaling, const float K[4],
                         __nv_bfloat16 *feat, cudaStream_t s) {
  const size_t pix = (size_t)W * H;
  for (int i = 0; i < n; i += FEATURE_IMAGES_MAX) {
    FeatureImages images;
    const int m = std::min(n - i, FEATURE_IMAGES_MAX);
    for (int k = 0; k < m; k++) {
      images.depth[k] = depth + (size_t)(i + k) * pix;
      for (int c = 0; c < 4; c++) images.K[k][c] = K[c];
    }
    const cudaError_t e = cnn_features_of(images, m, W, H, scaling, feat + (size_t)i * pix * CNN_FEAT_CH, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t cnn_forward(const __nv_bfloat16 *params, const __nv_bfloat16 *feat, int n, int W, int H,
                        __nv_bfloat16 *a1, __nv_bfloat16 *a2, float *out, float tau_cm, uint32_t *err, int err_stride,
                        cudaStream_t s) {
  cudaError_t e = ensure_attrs();
  if (e != cudaSuccess) return e;
  conv<8, 16, CONV_RELU_BF16>(feat, n, W, H, params + P_W1, params + P_B1, a1, 0.0f, err, err_stride, s);
  conv<16, 16, CONV_RELU_BF16>(a1, n, W, H, params + P_W2, params + P_B2, a2, 0.0f, err, err_stride, s);
  if (tau_cm > 0.0f)
    conv<16, 1, CONV_CONF>(a2, n, W, H, params + P_W3, params + P_B3, out, 1.0f / tau_cm, err, err_stride, s);
  else
    conv<16, 1, CONV_F32>(a2, n, W, H, params + P_W3, params + P_B3, out, 0.0f, err, err_stride, s);
  return cudaGetLastError();
}

cudaError_t cnn_backward(const __nv_bfloat16 *params, const __nv_bfloat16 *feat, const __nv_bfloat16 *a1,
                         const __nv_bfloat16 *a2, const float *dpred, int n, int W, int H, float *g1, float *g2,
                         float *grads, cudaStream_t s) {
  cudaError_t e = ensure_attrs();
  if (e != cudaSuccess) return e;
  // layer 3
  if ((e = wgrad<WG_L3>(a2, dpred, n, W, H, grads + P_W3, grads + P_B3, s)) != cudaSuccess) return e;
  input_grad<RC_F32_1>(dpred, n, W, H, params + P_W3, g2, a2, s);
  // layer 2
  if ((e = wgrad<WG_L2>(a1, g2, n, W, H, grads + P_W2, grads + P_B2, s)) != cudaSuccess) return e;
  input_grad<RC_F32_16>(g2, n, W, H, params + P_W2, g1, a1, s);
  // layer 1 (no gradient of the input)
  if ((e = wgrad<WG_L1>(feat, g1, n, W, H, grads + P_W1, grads + P_B1, s)) != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t cnn_mse(const float *pred, const float *target, int64_t count, float inv_count, float *dpred,
                    double *loss, cudaStream_t s) {
  const int blocks = (int)std::min<int64_t>((count + 255) / 256, 148 * 8);
  note_launch();
  k_cnn_mse<<<std::max(blocks, 1), 256, 0, s>>>(pred, target, count, inv_count, dpred, loss);
  return cudaGetLastError();
}

cudaError_t cnn_adam(float *master, __nv_bfloat16 *params, float *grads, float *m, float *v, int n, float lr,
                     float b1, float b2, float eps, int step, cudaStream_t s) {
  const float bc1 = 1.0f - powf(b1, (float)step), bc2 = 1.0f - powf(b2, (float)step);
  note_launch();
  k_cnn_adam<<<(n + 255) / 256, 256, 0, s>>>(master, params, grads, m, v, n, lr, b1, b2, eps, bc1, bc2);
  return cudaGetLastError();
}

cudaError_t launch_raycast(const RaycastMap &m, const CamF &p, int W, int H, const uint16_t *depth, float scaling,
                           float window, float step, float *out, cudaStream_t s) {
  note_launch();
  k_raycast<<<dim3((W + RAY_W - 1) / RAY_W, (H + RAY_H - 1) / RAY_H), RAY_THREADS, 0, s>>>(m, p, W, H, depth, scaling, window, step, out);
  return cudaGetLastError();
}

}  // namespace ffb
