// Front-to-back alpha compositing, forward and backward (reference src/rasterize.rs).
//
// The forward gives every warp an 8x4 pixel sub-block of a tile, one pixel per lane in scalar
// arithmetic; the default backward an 8x8 one, two pixels per lane as f32x2 pairs. The tile's
// warps scan its sorted list together, 1,024 entries at a time with barriers around each scan,
// for the sub-blocks that an entry's pixel rectangle touches; every warp then walks the entries
// of its own sub-block alone, staging records in its own shared memory (32 at a time, 16 in the
// backward, gathered while the ones before are composited). The one-pixel-per-thread backward
// and the deterministic one stage chunks for the whole block. Tile shape (16x16 by default; 8x8
// and 16x32 too) and, for the one-pixel backward, chunk depth are template parameters chosen at
// run time from the context's configuration (the autotuner's pick). Every per-pixel decision
// (sigma range, alpha >= 1/255, the 0.99 clamp, T < 1e-4) is taken on values computed exactly as
// the reference computes them: unfused arithmetic and a correctly rounded exp.
#include <mutex>
#include <set>
#include <type_traits>
#include <utility>

#include "common.cuh"
#include "kernels.cuh"
#include "pair.cuh"

namespace splat {

// Geometry of a TW x TH tile: TW * TH threads, warps over 8x4 sub-blocks row by row. An
// entry's pixel rectangle within the tile is a column mask and a row mask packed in one
// word (rows from bit kRowShift), 32 bits while the rows fit in 16, else 64.
template <int TW, int TH>
struct TileGeo {
  static constexpr int kThreads = TW * TH;
  static constexpr int kWarps = kThreads / 32;
  static constexpr int kWarpsX = TW / 8;
  static constexpr int kRowShift = TH > 16 ? 32 : 16;
  typedef typename std::conditional<(TH > 16), unsigned long long, uint32_t>::type Mask;
  typedef typename std::conditional<(kWarps > 8), uint16_t, uint8_t>::type WarpMask;
  static_assert(TW % 8 == 0 && TH % 4 == 0 && TW <= 16 && TH <= 32, "tile shape");
};

// evaluate (rasterize.rs:231-244), scalar, with the general correctly rounded exp. Returns
// false when skipped.
__device__ __forceinline__ bool evaluate_ref(float px, float py, float mx, float my, float A, float B, float C,
                                             float opacity, float sigma_max, float* gauss_out, float* alpha_out) {
  const float dx = px - mx;
  const float dy = py - my;
  const float sigma = 0.5f * (A * dx * dx + C * dy * dy) + B * dx * dy;
  if (sigma < 0.0f || sigma > sigma_max) return false;
  const float gauss = crm::expf_cr(-sigma);
  const float og = opacity * gauss;
  if (og < SPLAT_ALPHA_MIN) return false;
  *gauss_out = gauss;
  *alpha_out = fminf(og, SPLAT_ALPHA_MAX);
  return true;
}

// evaluate for the backward pass. The decisions must be the forward's, which were taken on
// the correctly rounded exp; the value may carry a few ulps. A fast exp (MUFU ex2) decides
// whenever the product opacity * gauss lies outside a relative band of kExpBand around the
// two thresholds (1/255 and 0.99); inside the band the correctly rounded exp is evaluated
// and decides. kExpBand bounds the fast exp's relative error on the argument range
// [-ln(255), 0] with a wide margin (the bound is checked on the device by
// splat_diag_fast_exp_error). *unclamped is the reference's `opacity * gauss < 0.99`.
constexpr float kExpBand = 3e-5f;

// exp(x) through the special-function unit: 2^(x log2 e), the product rounded to nearest,
// then ex2.approx (flush-to-zero). Relative error of the product's rounding is 2^-24 of an
// exponent below 9 in magnitude on the range used, and ex2.approx's own is about 2^-22;
// splat_diag_fast_exp_error measures the sum on every float of the range.
constexpr float kLog2e = 1.44269504088896341f;

__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float fast_exp(float x) { return ex2_approx(__fmul_rn(x, kLog2e)); }

// sigma = 0.5 (A dx dx + C dy dy) + B dx dy for a pair of pixels, operation for operation as
// the reference (rasterize.rs:236), one rounding per operation (f2_mul is never contracted);
// cdyy = (C dy) dy.
__device__ __forceinline__ f2 paired_sigma(f2 A, f2 B, f2 dx, f2 dy, f2 cdyy) {
  return f2_add(f2_mul(f2_splat(0.5f), f2_add(f2_mul(f2_mul(A, dx), dx), cdyy)), f2_mul(f2_mul(B, dx), dy));
}

__device__ __forceinline__ bool evaluate_bwd(float px, float py, float mx, float my, float A, float B, float C,
                                             float opacity, float sigma_max, float* gauss_out, float* alpha_out,
                                             bool* unclamped) {
  const float dx = px - mx;
  const float dy = py - my;
  const float sigma = 0.5f * (A * dx * dx + C * dy * dy) + B * dx * dy;
  if (sigma < 0.0f || sigma > sigma_max) return false;
  float gauss = fast_exp(-sigma);
  float og = opacity * gauss;
  const bool near_min = fabsf(og - SPLAT_ALPHA_MIN) < SPLAT_ALPHA_MIN * kExpBand;
  const bool near_max = fabsf(og - SPLAT_ALPHA_MAX) < SPLAT_ALPHA_MAX * kExpBand;
  if (near_min || near_max) {
    gauss = crm::expf_cr(-sigma);
    og = opacity * gauss;
  }
  if (og < SPLAT_ALPHA_MIN) return false;
  *gauss_out = gauss;
  *alpha_out = fminf(og, SPLAT_ALPHA_MAX);
  *unclamped = og < SPLAT_ALPHA_MAX;
  return true;
}

// Largest relative error of the fast exp against the correctly rounded one over every
// float in [lo, hi] (a diagnostic of the bound kExpBand relies on).
__global__ void diag_fast_exp_kernel(uint32_t lo_bits, uint32_t count, int negative, unsigned int* max_rel_bits) {
  float worst = 0.0f;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
    const uint32_t b = lo_bits + k;
    const float x = negative ? -__uint_as_float(b) : __uint_as_float(b);
    const float e = crm::expf_cr(x);
    const float f = fast_exp(x);
    if (e > 0.0f) worst = fmaxf(worst, fabsf(f - e) / e);
  }
  for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
  if ((threadIdx.x & 31) == 0) atomicMax(max_rel_bits, __float_as_uint(worst));
}

Status launch_diag_fast_exp(Ctx* c, float magnitude_lo, float magnitude_hi, int negative, float* out_host) {
  unsigned int* d = nullptr;
  SPLAT_TRY(arena_reserve(c, 4, (void**)&d));
  SPLAT_CUDA(cudaMemsetAsync(d, 0, 4, c->stream));
  const uint32_t lo = fbits(magnitude_lo), hi = fbits(magnitude_hi);
  diag_fast_exp_kernel<<<c->sm_count * 8, 256, 0, c->stream>>>(lo, hi - lo + 1, negative, d);
  c->launches.count++;
  SPLAT_LAUNCHED("diag_fast_exp_kernel");
  unsigned int h = 0;
  SPLAT_CUDA(cudaMemcpyAsync(&h, d, 4, cudaMemcpyDeviceToHost, c->stream));
  SPLAT_CUDA(cudaStreamSynchronize(c->stream));
  *out_host = bitsf(h);
  return Status::ok();
}

// Paired arithmetic against scalar unfused arithmetic on seeded inputs: [0] counts pixels
// whose paired_sigma differs from the scalar sigma of rasterize.rs:236, [1] blur steps
// acc + w x (the SSIM loss's accumulation) that differ. Both must be zero.
__device__ __forceinline__ float diag_uniform(uint32_t i, uint32_t salt, float lo, float hi) {
  uint32_t h = i * 0x9e3779b9u ^ salt;
  h ^= h >> 16;
  h *= 0x7feb352du;
  h ^= h >> 15;
  h *= 0x846ca68bu;
  h ^= h >> 16;
  return lo + (hi - lo) * (float)(h >> 8) * (1.0f / 16777216.0f);
}

__global__ void diag_pair_exact_kernel(uint32_t n, unsigned int* __restrict__ mism) {
  unsigned int bad_sigma = 0, bad_blur = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float A = diag_uniform(i, 1u, 0.0f, 3.4f), B = diag_uniform(i, 2u, -1.7f, 1.7f);
    const float C = diag_uniform(i, 3u, 0.0f, 3.4f), dx = diag_uniform(i, 4u, -48.0f, 48.0f);
    const float dy0 = diag_uniform(i, 5u, -48.0f, 48.0f), dy1 = diag_uniform(i, 6u, -48.0f, 48.0f);
    const f2 dy2 = f2_make(dy0, dy1), cdyy = f2_mul(f2_mul(f2_splat(C), dy2), dy2);
    float p0, p1;
    f2_split(paired_sigma(f2_splat(A), f2_splat(B), f2_splat(dx), dy2, cdyy), p0, p1);
    const float dys[2] = {dy0, dy1}, ps[2] = {p0, p1};
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const float dy = dys[q];
      const float s = __fadd_rn(__fmul_rn(0.5f, __fadd_rn(__fmul_rn(__fmul_rn(A, dx), dx), __fmul_rn(__fmul_rn(C, dy), dy))),
                                __fmul_rn(__fmul_rn(B, dx), dy));
      bad_sigma += !(ps[q] == s);
    }
    const float w = diag_uniform(i, 7u, 0.0f, 0.3f), acc0 = diag_uniform(i, 8u, -2.0f, 2.0f);
    const float acc1 = diag_uniform(i, 9u, 0.0f, 1.5f), x0 = diag_uniform(i, 10u, -0.2f, 1.2f);
    const float x1 = diag_uniform(i, 11u, 0.0f, 1.0f);
    float b0, b1;
    f2_split(f2_add(f2_make(acc0, acc1), f2_mul(f2_splat(w), f2_make(x0, x1))), b0, b1);
    bad_blur += !(b0 == __fadd_rn(acc0, __fmul_rn(w, x0))) + !(b1 == __fadd_rn(acc1, __fmul_rn(w, x1)));
  }
  for (int o = 16; o > 0; o >>= 1) {
    bad_sigma += __shfl_xor_sync(0xffffffffu, bad_sigma, o);
    bad_blur += __shfl_xor_sync(0xffffffffu, bad_blur, o);
  }
  if ((threadIdx.x & 31) == 0 && (bad_sigma | bad_blur)) {
    atomicAdd(&mism[0], bad_sigma);
    atomicAdd(&mism[1], bad_blur);
  }
}

Status launch_diag_pair_exact(Ctx* c, uint32_t n, uint32_t* out_host) {
  unsigned int* d = nullptr;
  SPLAT_TRY(arena_reserve(c, 8, (void**)&d));
  SPLAT_CUDA(cudaMemsetAsync(d, 0, 8, c->stream));
  diag_pair_exact_kernel<<<c->sm_count * 8, 256, 0, c->stream>>>(n, d);
  c->launches.count++;
  SPLAT_LAUNCHED("diag_pair_exact_kernel");
  SPLAT_CUDA(cudaMemcpyAsync(out_host, d, 8, cudaMemcpyDeviceToHost, c->stream));
  SPLAT_CUDA(cudaStreamSynchronize(c->stream));
  return Status::ok();
}

// The entry's pixel rectangle within the TW x TH tile whose top-left pixel is (ox, oy) as a
// mask of the columns (low bits) and a mask of the rows (from bit kRowShift) it covers.
template <int TW, int TH>
__device__ __forceinline__ typename TileGeo<TW, TH>::Mask tile_rect_masks(uint32_t rx, uint32_t ry, uint32_t ox,
                                                                           uint32_t oy) {
  typedef typename TileGeo<TW, TH>::Mask Mask;
  const int x0 = (int)(rx & 0xffffu) - (int)ox, x1 = (int)(rx >> 16) - (int)ox;
  const int y0 = (int)(ry & 0xffffu) - (int)oy, y1 = (int)(ry >> 16) - (int)oy;
  const uint32_t cx0 = (uint32_t)min(max(x0, 0), TW), cx1 = (uint32_t)min(max(x1, 0), TW);
  const uint32_t cy0 = (uint32_t)min(max(y0, 0), TH), cy1 = (uint32_t)min(max(y1, 0), TH);
  const uint32_t cols = cx1 > cx0 ? ((0xffffffffu >> (32u - (cx1 - cx0))) << cx0) : 0u;
  const uint32_t rows = cy1 > cy0 ? ((0xffffffffu >> (32u - (cy1 - cy0))) << cy0) : 0u;
  return (Mask)cols | ((Mask)rows << TileGeo<TW, TH>::kRowShift);
}

// Bit w of the result is set when the pixel rectangle (x0|x1<<16, y0|y1<<16, absolute
// pixels) overlaps warp w's 8 x SBH sub-block of the tile whose top-left pixel is (ox, oy)
// (warps row by row, TW / 8 across).
template <int TW, int TH, int SBH = 4>
__device__ __forceinline__ uint32_t subblock_mask(uint32_t rx, uint32_t ry, uint32_t ox, uint32_t oy) {
  constexpr int WX = TileGeo<TW, TH>::kWarpsX;
  const uint32_t x0 = rx & 0xffffu, x1 = rx >> 16, y0 = ry & 0xffffu, y1 = ry >> 16;
  bool col[WX];
#pragma unroll
  for (int qx = 0; qx < WX; qx++) col[qx] = x0 < ox + 8u * qx + 8u && x1 > ox + 8u * qx;
  uint32_t m = 0;
#pragma unroll
  for (uint32_t qy = 0; qy < (uint32_t)(TH / SBH); qy++) {
    const bool row = y0 < oy + (uint32_t)SBH * qy + (uint32_t)SBH && y1 > oy + (uint32_t)SBH * qy;
#pragma unroll
    for (int qx = 0; qx < WX; qx++)
      if (row && col[qx]) m |= 1u << (qy * WX + qx);
  }
  return m;
}

// Compacts, in order, the chunk-local indices k < cnt whose mask has this warp's bit (and,
// when `limit` is finite, k < limit) into list[]; returns how many.
template <typename WM>
__device__ __forceinline__ uint32_t build_warp_list(const WM* __restrict__ smask, uint32_t cnt, uint32_t limit,
                                                    uint8_t* __restrict__ list) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t n = 0;
  for (uint32_t b = 0; b < cnt; b += 32) {
    const uint32_t k = b + lane;
    const bool hit = k < cnt && k < limit && ((smask[k] >> warp) & 1u);
    const uint32_t bal = __ballot_sync(0xffffffffu, hit);
    if (hit) list[n + __popc(bal & lt)] = (uint8_t)k;
    n += __popc(bal);
  }
  __syncwarp();
  return n;
}

// ---------------------------------------------------------------------------------------
// A tile's list and the warps' walk of it, shared by the forward and the paired backward.
// ---------------------------------------------------------------------------------------
constexpr int kListChunk = 1024;  // list entries scanned at once: most tiles take one scan
constexpr int kStage = 32;        // entries staged per round, one per lane
constexpr int kQueue = 64;        // hits waiting to be staged: up to 31 + one step of 32

// Part of a tile's list in shared memory: every entry's Gaussian and the sub-blocks of the
// tile its pixel rectangle touches (one bit each).
template <typename Mask>
struct TileList {
  uint32_t g[kListChunk];
  Mask mask[kListChunk];
};

// Geometry of one warp's 8 x BH pixel sub-block: kPerTile warps share a tile.
template <int TW, int TH, int BH>
struct Walk {
  static constexpr int kPerTile = TW * TH / (8 * BH), kAcross = TW / 8;
  typedef typename std::conditional<(kPerTile > 8), uint16_t, uint8_t>::type Mask;

  uint32_t bx, by, ox, oy, width, height, sub;  // sub-block and tile origin, the view's size
  size_t pix0;                                  // the view's first pixel
  uint2 range;                                  // the tile's entries
  const uint32_t* gauss;
  const float4* rec;

  // Sub-block of warp `w` of the grid; false past the last tile (then for all its warps). A
  // batch numbers its tiles across the views.
  __device__ __forceinline__ bool init(uint32_t w, uint32_t tiles, uint32_t width_, uint32_t height_,
                                       uint32_t tiles_x, const uint32_t* __restrict__ gauss_,
                                       const float4* __restrict__ rec_, const uint2* __restrict__ ranges,
                                       const BatchTable* __restrict__ bt) {
    const uint32_t global = w / kPerTile;
    sub = w % kPerTile;
    if (global >= (bt ? bt->tile_start[bt->views] : tiles)) return false;
    uint32_t tile = global;
    pix0 = 0;
    width = width_;
    height = height_;
    if (bt) {
      const int v = batch_view_of(bt->tile_start, bt->views, global);
      tile = global - bt->tile_start[v];
      width = bt->cam[v].width;
      height = bt->cam[v].height;
      tiles_x = bt->tiles_x[v];
      pix0 = bt->pix_start[v];
    }
    ox = (tile % tiles_x) * TW;
    oy = (tile / tiles_x) * TH;
    bx = ox + (sub % kAcross) * 8u;
    by = oy + (sub / kAcross) * BH;
    range = ranges[global];
    gauss = gauss_ + range.x;
    rec = rec_;
    return true;
  }

  // Barrier over the tile's warps; a block holds `kTiles` tiles, each with a barrier of its own.
  template <int kTiles>
  __device__ __forceinline__ void barrier() const {
    if (kPerTile == 1) {
      __syncwarp();
    } else if (kTiles == 1) {
      __syncthreads();
    } else {
      const uint32_t id = 1u + (threadIdx.x >> 5) / kPerTile;
      asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "n"(32 * kPerTile) : "memory");
    }
  }
  // The same; true when `p` holds in every thread of the tile's warps.
  template <int kTiles>
  __device__ __forceinline__ bool barrier_all(bool p) const {
    if (kPerTile == 1) return __all_sync(0xffffffffu, p);
    if (kTiles == 1) return __syncthreads_and(p);
    const uint32_t id = 1u + (threadIdx.x >> 5) / kPerTile;
    uint32_t r;
    asm volatile(
        "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.and.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(id), "n"(32 * kPerTile)
        : "memory");
    return r != 0;
  }

  // The tile's warps scan list entries first, first + step, ... (`cnt` of them, step 1 or -1)
  // into `list`: each entry's rectangle is loaded once for the whole tile.
  __device__ __forceinline__ void scan(TileList<Mask>& list, uint32_t first, int step, uint32_t cnt) const {
    constexpr uint32_t kThreads = 32 * kPerTile, kBatch = kPerTile >= 8 ? kListChunk / kThreads : 4;
    const uint32_t t = sub * 32u + (threadIdx.x & 31u);
    for (uint32_t i0 = t; i0 < cnt; i0 += kThreads * kBatch) {
      uint32_t g[kBatch];
      float2 r[kBatch];
#pragma unroll
      for (uint32_t q = 0; q < kBatch; q++) {
        const uint32_t i = i0 + q * kThreads;
        g[q] = i < cnt ? gauss[first + (uint32_t)(step * (int)i)] : 0u;
      }
#pragma unroll
      for (uint32_t q = 0; q < kBatch; q++)
        if (i0 + q * kThreads < cnt) r[q] = reinterpret_cast<const float2*>(rec + 4 * (size_t)g[q] + 2)[1];
#pragma unroll
      for (uint32_t q = 0; q < kBatch; q++) {
        const uint32_t i = i0 + q * kThreads;
        if (i < cnt) {
          list.g[i] = g[q];
          list.mask[i] = (Mask)subblock_mask<TW, TH, BH>(fbits(r[q].x), fbits(r[q].y), ox, oy);
        }
      }
    }
  }
};

__device__ __forceinline__ void copy_async16(float4* smem, const float4* global) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(global) : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One warp's pass over a scanned list: the entries from `first` on whose mask has the warp's bit,
// in order, queued (as list indices) and staged STAGE (at most 32) at a time.
template <typename Mask, int STAGE>
struct Stager {
  const TileList<Mask>* list;
  uint32_t cnt, pos, head, tail, bit;
  uint16_t* queue;
  __device__ __forceinline__ void start(const TileList<Mask>* l, uint32_t first, uint32_t cnt_, uint32_t bit_,
                                        uint16_t* q) {
    list = l;
    cnt = cnt_;
    bit = bit_;
    queue = q;
    pos = first;
    head = tail = 0;
  }
  // Starts the copies of the next stage's records, part p of entry i to s + p * stride + i
  // (four lanes per record: one 64-byte line each); returns how many entries, and through *g
  // and *index this lane's Gaussian and list index.
  __device__ __forceinline__ uint32_t fetch(const float4* __restrict__ rec, float4* s, uint32_t stride, uint32_t* g,
                                            uint32_t* index) {
    const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    while (tail - head < (uint32_t)STAGE && pos < cnt) {
      const uint32_t i = pos + lane;
      const bool hit = i < cnt && ((list->mask[i] >> bit) & 1u);
      const uint32_t bal = __ballot_sync(0xffffffffu, hit);
      if (hit) queue[(tail + __popc(bal & lt)) & (kQueue - 1)] = (uint16_t)i;
      tail += __popc(bal);
      pos += 32u;
    }
    __syncwarp();
    const uint32_t m = min(tail - head, (uint32_t)STAGE);
    if (lane < m) {
      *index = queue[(head + lane) & (kQueue - 1)];
      *g = list->g[*index];
    }
    const uint32_t part = lane & 3u;
#pragma unroll
    for (uint32_t q = 0; q < STAGE / 8; q++) {
      const uint32_t i = 8u * q + (lane >> 2);
      const uint32_t gi = __shfl_sync(0xffffffffu, *g, i);
      if (i < m && part < 3u) copy_async16(s + part * stride + i, rec + 4 * (size_t)gi + part);
    }
    head += m;
    __syncwarp();
    return m;
  }
};

// 32x32 bit-matrix transpose across a warp: lane j holds row j on entry; on return lane L
// holds column L (bit j of the result = bit L of lane j's input). Five exchange stages,
// each swapping the off-diagonal blocks of size s.
__device__ __forceinline__ uint32_t warp_transpose_bits(uint32_t x) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t masks[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int i = 0; i < 5; i++) {
    const uint32_t sh = 16u >> i, m = masks[i];
    const uint32_t y = __shfl_xor_sync(0xffffffffu, x, sh);
    x = (lane & sh) ? ((x & ~m) | ((y & ~m) >> sh)) : ((x & m) | ((y & m) << sh));
  }
  return x;
}

// Columns (bits 0-7) and rows (bits 8-15) of the 8 x 8 block at (bx, by) inside the pixel
// rectangle (x0|x1<<16, y0|y1<<16); 0 in either half when it is empty.
__device__ __forceinline__ uint32_t sub_block_mask(uint32_t rx, uint32_t ry, uint32_t bx, uint32_t by) {
  const int x0 = min(max((int)(rx & 0xffffu) - (int)bx, 0), 8), x1 = min(max((int)(rx >> 16) - (int)bx, 0), 8);
  const int y0 = min(max((int)(ry & 0xffffu) - (int)by, 0), 8), y1 = min(max((int)(ry >> 16) - (int)by, 0), 8);
  const uint32_t cols = ((1u << x1) - 1u) & ~((1u << x0) - 1u);
  const uint32_t rows = ((1u << y1) - 1u) & ~((1u << y0) - 1u);
  return cols | (rows << 8);
}

// An entry whose sigma could overflow to inf or NaN, whose sigma_max passes the exp table or
// whose colour or opacity is not finite (none of which a projection of finite parameters
// gives) is composited by the scalar path.
__device__ __forceinline__ bool special_entry(float4 r0, float4 r1, float4 r2) {
  const bool plain = fabsf(r0.x) < 1e9f && fabsf(r0.y) < 1e9f && fabsf(r0.z) < 1e15f && fabsf(r0.w) < 1e15f &&
                     fabsf(r1.x) < 1e15f && fabsf(r1.y) < 1e15f && r1.z <= crm::kExpGridMax && fabsf(r1.w) < 1e30f &&
                     fabsf(r2.x) < 1e30f && fabsf(r2.y) < 1e30f;
  return !plain;
}

// forward_tile (rasterize.rs:249-302): each warp composites an 8x4 sub-block, one pixel per
// lane, entries in list (depth) order. For every 32 staged entries the coverage masks
// (lane j: the sub-block's pixels inside entry j's rectangle) are transposed across the warp,
// and each lane then walks only the entries that cover its own pixel, so the warp runs as
// many rounds as its busiest lane. A round has no branch on the decisions: a lane out of
// entries takes the null entry (index kStage), a pixel that skips its entry takes alpha = 0,
// which leaves transmittance and colour exactly as they are. exp is the correctly rounded one
// (crm::expf_cr_grid; its table in shared memory, six double operations). kCount adds the
// evaluated-pair counter (untimed diagnostics only).
// Bound by instruction issue (73%) and shared-memory reads (62%: divergent 16-byte record
// reads and the exp table). Time against one block per tile staging chunks between barriers,
// with a 577-entry exp table and its rounding in double: 1M Gaussians at 1920x1080 542 ->
// 428 us, 187k clustered at 1297x840 264 -> 194, 34k at 256x256 86 -> 53. 32 warps per SM (64
// registers) beat 40 (spills; 432, 199 and 60 us). A pixel pair per lane in f32x2 arithmetic
// with every lane on the same entry was slower on small Gaussians (616 us) and at 256x256.
struct FwdStage {
  float4 s[2][3][kStage + 1];  // records (three of their four quads), double-buffered; the last entry is null
  uint16_t queue[kQueue];
};
template <int TW, int TH>
struct FwdShape {
  typedef Walk<TW, TH, 4> W;
  static constexpr int kWarps = W::kPerTile > 8 ? W::kPerTile : 8, kTiles = kWarps / W::kPerTile;
};
template <int TW, int TH>
struct FwdSmem {
  double tab[crm::kExpGridEntries];
  FwdStage stage[FwdShape<TW, TH>::kWarps];
  TileList<typename Walk<TW, TH, 4>::Mask> list[FwdShape<TW, TH>::kTiles];
};

__device__ const crm::ExpGrid kExpGrid{};

template <int TW, int TH, bool kCount>
__global__ void __launch_bounds__(32 * FwdShape<TW, TH>::kWarps, 32 / FwdShape<TW, TH>::kWarps) raster_fwd_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ gauss, const uint2* __restrict__ ranges,
    uint32_t tiles, uint32_t width, uint32_t height, uint32_t tiles_x, float bg0, float bg1, float bg2,
    float* __restrict__ image, float* __restrict__ final_t, uint32_t* __restrict__ n_contrib,
    unsigned long long* __restrict__ pairs, const BatchTable* __restrict__ bt) {
  typedef FwdShape<TW, TH> Shape;
  typedef typename Shape::W W;
  extern __shared__ __align__(16) unsigned char raster_smem[];
  FwdSmem<TW, TH>& sm = *reinterpret_cast<FwdSmem<TW, TH>*>(raster_smem);
  for (int i = threadIdx.x; i < crm::kExpGridEntries; i += 32 * Shape::kWarps) sm.tab[i] = kExpGrid.v[i];
  chain_wait();  // the table is constant: it loads while the predecessor drains
  __syncthreads();
  const double* tab = sm.tab;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  W wk;
  if (!wk.init(blockIdx.x * Shape::kWarps + warp, tiles, width, height, tiles_x, gauss, rec, ranges, bt)) return;
  FwdStage& st = sm.stage[warp];
  TileList<typename W::Mask>& list = sm.list[warp / W::kPerTile];
  if (lane < 2) {
    st.s[lane][0][kStage] = st.s[lane][2][kStage] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    st.s[lane][1][kStage] = make_float4(0.0f, 0.0f, -1.0f, 0.0f);  // sigma_max < 0: never taken
  }
  const uint32_t x = wk.bx + (lane & 7u), y = wk.by + (lane >> 3);
  const bool inside = x < wk.width && y < wk.height;
  const float px = (float)x + 0.5f, py = (float)y + 0.5f;
  float T = 1.0f, cr = 0.0f, cg = 0.0f, cb = 0.0f;
  uint32_t ncon = 0, npairs = 0;
  bool done = !inside;

  const uint32_t n = wk.range.y - wk.range.x;
  for (uint32_t first = 0; first < n; first += kListChunk) {
    if (first && wk.template barrier_all<Shape::kTiles>(done)) break;
    const uint32_t cnt = min(n - first, (uint32_t)kListChunk);
    wk.scan(list, first, 1, cnt);
    wk.template barrier<Shape::kTiles>();
    if (__all_sync(0xffffffffu, done)) continue;
    Stager<typename W::Mask, kStage> stager;
    stager.start(&list, 0, cnt, wk.sub, st.queue);
    uint32_t buf = 0, g = 0, index = 0;
    uint32_t m = stager.fetch(rec, st.s[0][0], kStage + 1, &g, &index);
    while (m) {
      copy_async_wait();
      __syncwarp();
      const float4* s0 = st.s[buf][0];
      const float4* s1 = st.s[buf][1];
      const float4* s2 = st.s[buf][2];
      uint32_t cov = 0;
      bool special = false;
      if (lane < m) {
        const float4 r2 = s2[lane];
        const uint32_t mask = sub_block_mask(fbits(r2.z), fbits(r2.w), wk.bx, wk.by);
        const uint32_t r4 = (mask >> 8) & 0xfu;
        cov = (mask & 0xffu) * ((r4 & 1u) | ((r4 & 2u) << 7) | ((r4 & 4u) << 14) | ((r4 & 8u) << 21));
        special = special_entry(s0[lane], s1[lane], r2);
      }
      const uint32_t place = first + index + 1u;  // n_contrib of a pixel whose last entry is this lane's
      special = __any_sync(0xffffffffu, special);
      uint32_t mine = warp_transpose_bits(cov);
      if (done) mine = 0;
      buf ^= 1u;
      m = stager.fetch(rec, st.s[buf][0], kStage + 1, &g, &index);  // loads while this stage is composited
      if (kCount) npairs += __popc(mine);
      uint32_t taken = kStage;  // the stage's last entry this pixel took
      if (!special) {
        while (__any_sync(0xffffffffu, mine != 0u)) {
          const uint32_t k = mine ? (uint32_t)__ffs((int)mine) - 1u : (uint32_t)kStage;
          mine &= mine - 1u;
          const float4 e0 = s0[k], e1 = s1[k];
          const float2 e2 = *reinterpret_cast<const float2*>(s2 + k);
          const float dx = px - e0.x, dy = py - e0.y;
          const float sigma = 0.5f * (e0.z * dx * dx + e1.x * dy * dy) + e0.w * dx * dy;
          const bool in = sigma >= 0.0f && sigma <= e1.z;
          const float og = e1.y * crm::expf_cr_grid(in ? sigma : crm::kExpGridSkip, tab);
          float alpha = og < SPLAT_ALPHA_MIN ? 0.0f : fminf(og, SPLAT_ALPHA_MAX);
          float test_t = T * (1.0f - alpha);
          if (test_t < SPLAT_T_MIN) {  // the pixel is done without this entry
            if (kCount) npairs -= __popc(mine);
            done = true;
            mine = 0;
            alpha = 0.0f;
            test_t = T;
          }
          const float at = alpha * T;
          cr += at * e1.w;
          cg += at * e2.x;
          cb += at * e2.y;
          T = test_t;
          taken = alpha > 0.0f ? k : taken;
        }
      } else {
        while (mine) {
          const uint32_t k = (uint32_t)__ffs((int)mine) - 1u;
          mine &= mine - 1u;
          const float4 e0 = s0[k], e1 = s1[k], e2 = s2[k];
          float gval, alpha;
          if (!evaluate_ref(px, py, e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, &gval, &alpha)) continue;
          const float test_t = T * (1.0f - alpha);
          if (test_t < SPLAT_T_MIN) {
            if (kCount) npairs -= __popc(mine);
            done = true;
            break;
          }
          const float at = alpha * T;
          cr += at * e1.w;
          cg += at * e2.x;
          cb += at * e2.y;
          T = test_t;
          taken = k;
        }
      }
      const uint32_t last_place = __shfl_sync(0xffffffffu, place, taken & 31u);
      if (taken < (uint32_t)kStage) ncon = last_place;
      if (__all_sync(0xffffffffu, done)) break;
    }
    copy_async_wait();  // copies may be in flight past an early stop
    __syncwarp();
  }
  if (inside) {
    const size_t pix = wk.pix0 + (size_t)y * wk.width + x;
    image[3 * pix] = cr + T * bg0;
    image[3 * pix + 1] = cg + T * bg1;
    image[3 * pix + 2] = cb + T * bg2;
    final_t[pix] = T;
    n_contrib[pix] = ncon;
  }
  if (kCount) {
    unsigned long long np = npairs;
    for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
    if (lane == 0 && np) atomicAdd(pairs, np);
  }
}

// backward_tile (rasterize.rs:354-455) for one tile per block. Per-pixel contributions to
// an entry's 11 gradient slots are summed across the warp by a transposing butterfly
// (13 shuffles leave each slot's warp total in a pair of lanes), across the block's warps
// with one shared-memory atomic instruction per warp, and across tiles with three float4
// vector atomics per entry.
// Slots per entry: ProjGrad (9), the AbsGS accumulators (2) and the entry's blending weight
// sum(alpha * T) over the tile's pixels (the trainer's contribution statistic).
constexpr int kSlots = 12;

// v[0..11] per lane in; out, the warp total of slot 6*b4 + 3*b3 + 2*b2 + b1 (b_i = bit i of
// the lane) when 2*b2 + b1 < 3, in both lanes of a pair. Each exchange stage keeps the half
// of the values selected by the lane's bit and adds the partner's copy of that half:
// 6 + 3 + 2 + 1 + 1 = 13 shuffles for 12 slots.
__device__ __forceinline__ float warp_transpose_reduce12(const float v[12]) {
  const uint32_t lane = threadIdx.x & 31;
  const bool b4 = lane & 16u, b3 = lane & 8u, b2 = lane & 4u, b1 = lane & 2u;
  float w[6], x[4], y[2];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    const float send = b4 ? v[i] : v[i + 6];
    const float keep = b4 ? v[i + 6] : v[i];
    w[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
  }
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float send = b3 ? w[i] : w[i + 3];
    const float keep = b3 ? w[i + 3] : w[i];
    x[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
  }
  x[3] = 0.0f;
#pragma unroll
  for (int i = 0; i < 2; i++) {
    const float send = b2 ? x[i] : x[i + 2];
    const float keep = b2 ? x[i + 2] : x[i];
    y[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
  }
  const float send = b1 ? y[0] : y[1];
  const float keep = b1 ? y[1] : y[0];
  float z = keep + __shfl_xor_sync(0xffffffffu, send, 2);
  z += __shfl_xor_sync(0xffffffffu, z, 1);
  return z;
}

// 1 / x for x in [0.01, 1] by the special-function unit alone (relative error within a few
// ulps; values only, never a decision). Over a pixel's reverse walk the recovered
// transmittance then carries at most about one ulp per entry walked, far inside the
// gradients' 1e-3 bar.
__device__ __forceinline__ float rcp_fast(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// PPL pixels per thread in scalar arithmetic: a warp owns an 8 x (4 PPL) sub-block, lane L
// the pixels (L % 8, L / 8 + 4 q) of it for q < PPL. It is launched with one pixel per
// thread (64 registers, 32 warps per SM); two pixels per thread run as pairs in
// raster_bwd_x2_kernel below, which replaced this kernel's PPL = 2 form (1.24-1.27 ms
// against 0.91 ms on the render benchmark).
template <int TW, int TH, int CH, int PPL>
__global__ void __launch_bounds__(TW * TH / PPL, (PPL == 1 ? 1024 : 768) / (TW * TH / PPL)) raster_bwd_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ gauss, const uint2* __restrict__ ranges,
    uint32_t width, uint32_t height, uint32_t tiles_x, float bg0, float bg1, float bg2,
    const float* __restrict__ final_t, const uint32_t* __restrict__ n_contrib, const float* __restrict__ dimage,
    float4* __restrict__ pgrad, int64_t cap, unsigned long long* __restrict__ pairs,
    const BatchTable* __restrict__ bt) {
  chain_wait();
  typedef TileGeo<TW, TH> Geo;
  constexpr int NT = TW * TH / PPL, NW = NT / 32, WX = TW / 8, SBH = 4 * PPL;
  typedef typename std::conditional<(NW > 8), uint16_t, uint8_t>::type WarpMask;
  if (bt && blockIdx.x >= bt->tile_start[bt->views]) return;  // past the batch's tiles
  __shared__ float4 s0[CH], s1[CH];
  __shared__ float2 s2[CH];
  __shared__ typename Geo::Mask srect[CH];
  __shared__ uint32_t sg[CH];
  __shared__ float acc[CH * kSlots];
  __shared__ WarpMask smask[CH];
  __shared__ uint8_t slist[NW][CH];
  __shared__ uint32_t s_max_last;
  // In a batch the block is a global tile: find its view, local tile and image offset.
  uint32_t tile = blockIdx.x;
  size_t pix0 = 0;
  if (bt) {
    const int v = batch_view_of(bt->tile_start, bt->views, blockIdx.x);
    tile = blockIdx.x - bt->tile_start[v];
    width = bt->cam[v].width;
    height = bt->cam[v].height;
    tiles_x = bt->tiles_x[v];
    pix0 = bt->pix_start[v];
  }
  const uint32_t ox = (tile % tiles_x) * TW, oy = (tile / tiles_x) * TH;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t lx = (warp % WX) * 8u + (lane & 7u);        // column in the tile
  const uint32_t ly0 = (warp / WX) * (uint32_t)SBH + (lane >> 3);  // row of pixel 0 in the tile
  const float px = (float)(ox + lx) + 0.5f;
  const uint2 range = ranges[blockIdx.x];
  uint8_t* list = slist[warp];
  const uint32_t list_len = range.y - range.x;

  // Per pixel: contributor count, transmittance, dL/dpixel and the running sums of the
  // reverse walk (rasterize.rs:347-455).
  uint32_t last[PPL];
  // nbg = -T_final (bg . dL/dpixel): the background's share of dL/dalpha is nbg / (1 - alpha).
  float T[PPL], nbg[PPL], d0[PPL], d1[PPL], d2[PPL], py[PPL];
  float acc_r[PPL], acc_g[PPL], acc_b[PPL], last_alpha[PPL], lc_r[PPL], lc_g[PPL], lc_b[PPL];
  uint32_t lane_last = 0;
#pragma unroll
  for (int q = 0; q < PPL; q++) {
    const uint32_t y = oy + ly0 + 4u * q, x = ox + lx;
    py[q] = (float)y + 0.5f;
    last[q] = 0;
    T[q] = 1.0f;
    d0[q] = d1[q] = d2[q] = nbg[q] = 0.0f;
    if (x < width && y < height) {
      const size_t pix = pix0 + (size_t)y * width + x;
      last[q] = min(n_contrib[pix], list_len);  // n_contrib never exceeds its tile's list
      T[q] = final_t[pix];
      d0[q] = dimage[3 * pix];
      d1[q] = dimage[3 * pix + 1];
      d2[q] = dimage[3 * pix + 2];
      nbg[q] = -T[q] * (bg0 * d0[q] + bg1 * d1[q] + bg2 * d2[q]);
    }
    acc_r[q] = acc_g[q] = acc_b[q] = 0.0f;  // accum (rasterize.rs:347)
    last_alpha[q] = lc_r[q] = lc_g[q] = lc_b[q] = 0.0f;
    lane_last = max(lane_last, last[q]);
  }
  if (threadIdx.x == 0) s_max_last = 0;
  for (int i = threadIdx.x; i < CH * kSlots; i += NT) acc[i] = 0.0f;
  __syncthreads();
  const uint32_t warp_max_last = __reduce_max_sync(0xffffffffu, lane_last);
  if (lane == 0) atomicMax(&s_max_last, warp_max_last);
  __syncthreads();
  const uint32_t max_last = s_max_last;
  uint32_t npairs = 0;

  for (uint32_t cend = max_last; cend > 0;) {
    const uint32_t cstart = cend > (uint32_t)CH ? cend - CH : 0u;
    const uint32_t cnt = cend - cstart;
#pragma unroll
    for (uint32_t e = threadIdx.x; e < (uint32_t)CH; e += NT) {
      uint32_t m = 0;
      if (e < cnt) {
        const uint32_t g = gauss[range.x + cstart + e];
        sg[e] = g;
        s0[e] = rec[4 * (size_t)g];
        s1[e] = rec[4 * (size_t)g + 1];
        const float4 e2 = rec[4 * (size_t)g + 2];
        s2[e] = make_float2(e2.x, e2.y);
        srect[e] = tile_rect_masks<TW, TH>(fbits(e2.z), fbits(e2.w), ox, oy);
        m = subblock_mask<TW, TH, SBH>(fbits(e2.z), fbits(e2.w), ox, oy);
      }
      smask[e] = (WarpMask)m;
    }
    __syncthreads();
    // Entries at or past every lane's n_contrib contribute nothing to this warp.
    const uint32_t limit = warp_max_last > cstart ? warp_max_last - cstart : 0u;
    const uint32_t nl = build_warp_list(smask, cnt, limit, list);
    for (int i = (int)nl - 1; i >= 0; i--) {
      const uint32_t kk = list[i];
      const uint32_t k = cstart + kk;
      const typename Geo::Mask rm = srect[kk];
      float c[kSlots];
#pragma unroll
      for (int q = 0; q < kSlots; q++) c[q] = 0.0f;
      bool active = false;
      const bool col_in = (uint32_t)(rm >> lx) & 1u;
#pragma unroll
      for (int q = 0; q < PPL; q++) {
        if (!(col_in && k < last[q] && ((uint32_t)(rm >> (ly0 + 4u * q + Geo::kRowShift)) & 1u))) continue;
        const float2 e2 = s2[kk];
        npairs++;
        const float4 e0 = s0[kk], e1 = s1[kk];
        float gval, alpha;
        bool unclamped;
        if (!evaluate_bwd(px, py[q], e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, &gval, &alpha, &unclamped)) continue;
        active = true;
        // Values only from here on: the arithmetic is fused and the divisions are
        // reciprocals; every decision was taken above exactly as in the forward pass.
        const float col_r = e1.w, col_g = e2.x, col_b = e2.y;
        const float inv = rcp_fast(1.0f - alpha);
        T[q] = T[q] * inv;
        const float t = T[q];
        const float keep = 1.0f - last_alpha[q];
        acc_r[q] = __fmaf_rn(last_alpha[q], lc_r[q], keep * acc_r[q]);
        acc_g[q] = __fmaf_rn(last_alpha[q], lc_g[q], keep * acc_g[q]);
        acc_b[q] = __fmaf_rn(last_alpha[q], lc_b[q], keep * acc_b[q]);
        float dalpha = (col_r - acc_r[q]) * d0[q];
        dalpha = __fmaf_rn(col_g - acc_g[q], d1[q], dalpha);
        dalpha = __fmaf_rn(col_b - acc_b[q], d2[q], dalpha);
        const float at = alpha * t;
        c[6] = __fmaf_rn(at, d0[q], c[6]);
        c[7] = __fmaf_rn(at, d1[q], c[7]);
        c[8] = __fmaf_rn(at, d2[q], c[8]);
        c[11] += at;
        lc_r[q] = col_r;
        lc_g[q] = col_g;
        lc_b[q] = col_b;
        last_alpha[q] = alpha;
        dalpha = __fmaf_rn(dalpha, t, nbg[q] * inv);
        if (unclamped) {
          const float opacity = e1.y;
          c[5] = __fmaf_rn(gval, dalpha, c[5]);
          const float dsigma = -(opacity * dalpha) * gval;
          const float dx = px - e0.x;
          const float dy = py[q] - e0.y;
          const float ddx = dsigma * __fmaf_rn(e0.z, dx, e0.w * dy);
          const float ddy = dsigma * __fmaf_rn(e0.w, dx, e1.x * dy);
          c[0] -= ddx;
          c[1] -= ddy;
          const float hs = 0.5f * dsigma;
          c[2] = __fmaf_rn(hs * dx, dx, c[2]);
          c[3] = __fmaf_rn(dsigma * dx, dy, c[3]);
          c[4] = __fmaf_rn(hs * dy, dy, c[4]);
          c[9] += fabsf(ddx);
          c[10] += fabsf(ddy);
        }
      }
      if (__any_sync(0xffffffffu, active)) {
        const float tot = warp_transpose_reduce12(c);
        const uint32_t local = (lane >> 1) & 3u;
        const uint32_t slot = 6u * ((lane >> 4) & 1u) + 3u * ((lane >> 3) & 1u) + local;
        if (!(lane & 1u) && local < 3u) atomicAdd(&acc[kk * kSlots + slot], tot);
      }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t e = threadIdx.x; e < (uint32_t)CH; e += NT) {
      if (e >= cnt) break;
      float* a = &acc[e * kSlots];
      const size_t g = sg[e];
      const float4 v0 = make_float4(a[0], a[1], a[2], a[3]);
      const float4 v1 = make_float4(a[4], a[5], a[6], a[7]);
      const float4 v2 = make_float4(a[8], a[9], a[10], a[11]);
      if (v0.x != 0.0f || v0.y != 0.0f || v0.z != 0.0f || v0.w != 0.0f) atomicAdd(&pgrad[g], v0);
      if (v1.x != 0.0f || v1.y != 0.0f || v1.z != 0.0f || v1.w != 0.0f) atomicAdd(&pgrad[cap + g], v1);
      if (v2.x != 0.0f || v2.y != 0.0f || v2.z != 0.0f || v2.w != 0.0f) atomicAdd(&pgrad[2 * cap + g], v2);
#pragma unroll
      for (int q = 0; q < kSlots; q++) a[q] = 0.0f;
    }
    __syncthreads();
    cend = cstart;
  }
  if (pairs) {
    unsigned long long np = npairs;
    for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
    if (lane == 0 && np) atomicAdd(pairs, np);
  }
}

// Backward decisions without the exp. The reference skips a pixel when sigma < 0, sigma >
// sigma_max or fl(opacity * exp(-sigma)) < 1/255 (rasterize.rs:231-244), with sigma_max =
// ln(opacity * 255) (both correctly rounded). fl(opacity * exp(-sigma)) does not increase
// with sigma, and for sigma <= sigma_max - kSigmaEdge it is at least
// (1/255) e^(kSigmaEdge - 7.2e-7) (1 - 2^-23) > 1/255 (the roundings of the quotient, the
// logarithm, the difference, the exp and the product, with ln(255 opacity) <= ln 255), so
// such a pixel passes the alpha test whatever the exp's value: the decision needs sigma
// only. Pixels within kSigmaEdge of sigma_max take the correctly rounded exp. Likewise
// fl(opacity * exp(-sigma)) <= opacity, so an entry with opacity < 0.99 never clamps.
constexpr float kSigmaEdge = 1e-4f;

// The backward with two pixels per thread computed as pairs, each warp alone on an 8x8
// sub-block (pair p = the pixels (p % 8, p / 8) and (p % 8, p / 8 + 4)), eight entries at a time
// in three phases.
//
// 1. Lane (e, q) = (lane % 8, lane / 8) holds entry e in registers and evaluates it at the
//    eight pairs of row q: sigma (bit-identical to the scalar sigma), the decisions by sigma's
//    threshold (above) and gauss, 0 where the pixel does not take the entry. No operand but
//    the pixels' n_contrib comes from shared memory, and a row's products with dy are made
//    once.
// 2. Lane p walks the taken entries in reverse depth order for pair p: transmittance, colour
//    accumulator, dL/dalpha (backward_tile, rasterize.rs:394-454). A pixel the entry does not
//    reach has alpha = 0: its transmittance is multiplied by rcp(1) = 1 exactly, its colour
//    accumulator by 0 + 1, and its contributions are exactly zero. What a pixel contributes
//    to the entry's gradients is two numbers: h = gauss dL/dalpha and w = alpha T.
// 3. Lane (e, q) sums h {1, dx, dx^2} (dy and its products are constant over a row), w {1,
//    dL/dr, dL/dg, dL/db}, h (A dx + B dy, B dx + C dy) and its absolute values over its row; the
//    12 slots follow by linear combination (with -dsigma = opacity h), two exchange stages add
//    the entry's four lanes, and one float4 vector atomic per gradient plane adds them to global
//    memory. The mean's gradient is summed pixel by pixel, not as A sum(h dx) + B sum(h dy): for
//    an elongated, tilted Gaussian these two nearly cancel, which amplified the sums' rounding
//    (axes 50 and 0.1 pixels: 1.5 times the error of summing in the reference's order, now 0.7).
//
// The phases hand (gauss) and (h, w) over in two 8 x 32 arrays of pairs in shared memory.
// Against one pixel pair per lane for everything (records broadcast from shared memory with
// each scalar duplicated, a 13-shuffle reduction of 12 slots over the warp for every entry)
// this takes about 134 instead of 185 warp instructions per entry. Bound by latency and issue
// (62% of the issue slots, FMA pipe 52%, shared-memory accesses 56%; DRAM 5% of its peak).
// Time: 1M Gaussians at 1920x1080 975 -> 666 us, 187k clustered at 1297x840 377 -> 257, 34k at
// 256x256 164 -> 79, 20k wide ones at 1386x1080 163 -> 117. kCount adds the evaluated-pair
// counter (untimed diagnostics only).
constexpr int kGroup = 8;      // entries per round of the three phases
constexpr int kBwdStage = 16;  // entries staged per copy
constexpr int kPairRow = 33;   // pairs per row and a pad: 8 rows x 2 quarters hit 16 distinct bank pairs
struct BwdStage {
  float4 s[2][3][kBwdStage];     // staged records (three of their four quads), double-buffered
  float4 color[kGroup];          // (opacity, r, g, b)
  float2 h[kGroup][kPairRow];    // gauss, then h; then the sums on their way out
  float2 w[kGroup][kPairRow];
  float4 d01[32];                // dL/dr and dL/dg of a pair
  float2 d2[32];                 // dL/db
  uint2 last[32];                // n_contrib
  uint16_t queue[kQueue];
};
template <int TW, int TH>
struct BwdShape {
  typedef Walk<TW, TH, 8> W;
  static constexpr int kWarps = W::kPerTile > 4 ? W::kPerTile : 4, kTiles = kWarps / W::kPerTile;
};
template <int TW, int TH>
struct BwdSmem {
  BwdStage stage[BwdShape<TW, TH>::kWarps];
  TileList<typename Walk<TW, TH, 8>::Mask> list[BwdShape<TW, TH>::kTiles];
  uint32_t max_last[BwdShape<TW, TH>::kTiles];
};

// Whether the entry is decided pixel by pixel with the scalar rule: sigma could overflow to inf
// or NaN (never for a projection of finite parameters), or sigma_max is not a number or below
// kSigmaEdge.
__device__ __forceinline__ bool special_geometry(float4 r0, float4 r1) {
  const bool plain = fabsf(r0.x) < 1e9f && fabsf(r0.y) < 1e9f && fabsf(r0.z) < 1e15f && fabsf(r0.w) < 1e15f &&
                     fabsf(r1.x) < 1e15f && r1.z < 1e30f && r1.z >= kSigmaEdge;
  return !plain;
}

// Phase 1 of one lane: gauss of its entry at the eight pairs of row q into st.h[e], 0 where the
// pixel does not take it. kLast tests the pixels' n_contrib (not needed when the entry is
// ahead of all of them).
template <bool kCount, bool kLast>
__device__ __forceinline__ void evaluate_row(BwdStage& st, uint32_t e, uint32_t q, float px0, float4 r0, f2 dy,
                                             f2 cdyy, uint32_t mask, uint32_t place, float sure, uint32_t sure_bits,
                                             uint32_t& nearest, f2& sum, uint32_t& npairs) {
  const f2 A = f2_splat(r0.z), B = f2_splat(r0.w), mx = f2_splat(r0.x), one = f2_splat(1.0f);
  const float inf = __int_as_float(0x7f800000);
  f2 px = f2_splat(px0);
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const f2 dx = f2_sub(px, mx);
    px = f2_add(px, one);
    const f2 sigma = paired_sigma(A, B, dx, dy, cdyy);
    float s0, s1, t0, t1;
    f2_split(sigma, s0, s1);
    f2_split(f2_sub(sigma, f2_splat(sure)), t0, t1);
    nearest = __vimin3_u32(nearest, fbits(t0), fbits(t1));
    bool in0 = (mask >> c) & 1u, in1 = in0;
    if (kLast) {
      const uint2 lp = st.last[8u * q + c];
      in0 = in0 && place < lp.x;
      in1 = in1 && place < lp.y;
    }
    if (kCount) {
      npairs += in0 && ((mask >> (8u + q)) & 1u);
      npairs += in1 && ((mask >> (12u + q)) & 1u);
    }
    const bool v0 = in0 && fbits(s0) <= sure_bits, v1 = in1 && fbits(s1) <= sure_bits;
    float g0, g1;
    f2_split(f2_mul(f2_make(v0 ? s0 : inf, v1 ? s1 : inf), f2_splat(-kLog2e)), g0, g1);
    g0 = ex2_approx(g0);
    g1 = ex2_approx(g1);
    st.h[e][8u * q + c] = make_float2(g0, g1);  // fast exp
    sum = f2_add(sum, f2_make(g0, g1));
  }
}

// State of a lane's two pixels in the reverse walk.
struct PixelPair {
  f2 T, nbg, d0, d1, d2, acc_r, acc_g, acc_b;
};

// Phase 2 of a group: st.h holds gauss on entry and h on return, st.w alpha T. An
// entry that no pixel of the sub-block takes has gauss 0 and colour 0 and leaves the state as it
// is. First everything that does not depend on the state, for all entries at once, then the chain
// through it. kClamp: an opacity may reach 0.99, where alpha clamps and the gradients through
// sigma and opacity vanish (rasterize.rs:414-432). One branch-free body for eight entries: 677 -> 653
// us on 1M Gaussians at 1920x1080 against a branch around each entry (four entries at a time: no gain).
template <bool kClamp>
__device__ __forceinline__ void walk_entries(BwdStage& st, uint32_t lane, PixelPair& p) {
  f2 gauss[kGroup], alpha[kGroup], inv[kGroup];
#pragma unroll
  for (int k = 0; k < kGroup; k++) {
    const float2 g = st.h[k][lane];
    const float opacity = st.color[k].x;
    gauss[k] = f2_make(g.x, g.y);
    alpha[k] = f2_mul(f2_splat(opacity), gauss[k]);
    if (kClamp) {
      float a0, a1;
      f2_split(alpha[k], a0, a1);
      gauss[k] = f2_make(a0 < SPLAT_ALPHA_MAX ? g.x : 0.0f, a1 < SPLAT_ALPHA_MAX ? g.y : 0.0f);
      alpha[k] = f2_make(fminf(a0, SPLAT_ALPHA_MAX), fminf(a1, SPLAT_ALPHA_MAX));
    }
    // Values only from here on (fused, reciprocal for division).
    float o0, o1;
    f2_split(f2_sub(f2_splat(1.0f), alpha[k]), o0, o1);
    inv[k] = f2_make(rcp_fast(o0), rcp_fast(o1));
  }
#pragma unroll
  for (int k = 0; k < kGroup; k++) {
    const float4 color = st.color[k];
    p.T = f2_mul(p.T, inv[k]);
    const f2 dr = f2_sub(f2_splat(color.y), p.acc_r);
    const f2 dg = f2_sub(f2_splat(color.z), p.acc_g);
    const f2 db = f2_sub(f2_splat(color.w), p.acc_b);
    f2 dalpha = f2_fma(db, p.d2, f2_fma(dg, p.d1, f2_mul(dr, p.d0)));
    // The accumulator advances right after its use (accum + alpha (c - accum)): the operands
    // of the reference's update on the pixel's next entry.
    p.acc_r = f2_fma(alpha[k], dr, p.acc_r);
    p.acc_g = f2_fma(alpha[k], dg, p.acc_g);
    p.acc_b = f2_fma(alpha[k], db, p.acc_b);
    dalpha = f2_fma(dalpha, p.T, f2_mul(p.nbg, inv[k]));
    float2 h, w;
    f2_split(f2_mul(gauss[k], dalpha), h.x, h.y);
    f2_split(f2_mul(alpha[k], p.T), w.x, w.y);
    st.h[k][lane] = h;
    st.w[k][lane] = w;
  }
}

template <int TW, int TH, bool kCount, int kSmWarps>
__global__ void __launch_bounds__(32 * BwdShape<TW, TH>::kWarps, kSmWarps / BwdShape<TW, TH>::kWarps) raster_bwd_x2_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ gauss, const uint2* __restrict__ ranges,
    uint32_t tiles, uint32_t width, uint32_t height, uint32_t tiles_x, float bg0, float bg1, float bg2,
    const float* __restrict__ final_t, const uint32_t* __restrict__ n_contrib, const float* __restrict__ dimage,
    float4* __restrict__ pgrad, int64_t cap, unsigned long long* __restrict__ pairs,
    const BatchTable* __restrict__ bt) {
  chain_wait();
  typedef BwdShape<TW, TH> Shape;
  typedef typename Shape::W W;
  extern __shared__ __align__(16) unsigned char raster_smem[];
  BwdSmem<TW, TH>& sm = *reinterpret_cast<BwdSmem<TW, TH>*>(raster_smem);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  W wk;
  if (!wk.init(blockIdx.x * Shape::kWarps + warp, tiles, width, height, tiles_x, gauss, rec, ranges, bt)) return;
  BwdStage& st = sm.stage[warp];
  TileList<typename W::Mask>& list = sm.list[warp / W::kPerTile];
  uint32_t& tile_last = sm.max_last[warp / W::kPerTile];
  if (wk.sub == 0 && lane == 0) tile_last = 0;
  wk.template barrier<Shape::kTiles>();
  const uint32_t list_len = wk.range.y - wk.range.x;

  // Per pixel pair: contributor counts, transmittance, dL/dpixel, the background's share of
  // dL/dalpha (times 1 - alpha) and the colour accumulator.
  uint32_t last[2];
  float Tq[2], nbgq[2], d0q[2], d1q[2], d2q[2];
#pragma unroll
  for (int q = 0; q < 2; q++) {
    const uint32_t x = wk.bx + (lane & 7u), y = wk.by + (lane >> 3) + 4u * q;
    last[q] = 0;
    Tq[q] = 1.0f;
    d0q[q] = d1q[q] = d2q[q] = nbgq[q] = 0.0f;
    if (x < wk.width && y < wk.height) {
      const size_t pix = wk.pix0 + (size_t)y * wk.width + x;
      last[q] = min(n_contrib[pix], list_len);  // n_contrib never exceeds its tile's list
      Tq[q] = final_t[pix];
      d0q[q] = dimage[3 * pix];
      d1q[q] = dimage[3 * pix + 1];
      d2q[q] = dimage[3 * pix + 2];
      nbgq[q] = -Tq[q] * (bg0 * d0q[q] + bg1 * d1q[q] + bg2 * d2q[q]);
    }
  }
  PixelPair pp;
  pp.T = f2_make(Tq[0], Tq[1]);
  pp.nbg = f2_make(nbgq[0], nbgq[1]);
  pp.d0 = f2_make(d0q[0], d0q[1]);
  pp.d1 = f2_make(d1q[0], d1q[1]);
  pp.d2 = f2_make(d2q[0], d2q[1]);
  pp.acc_r = pp.acc_g = pp.acc_b = f2_splat(0.0f);
  st.d01[lane] = make_float4(d0q[0], d0q[1], d1q[0], d1q[1]);
  st.d2[lane] = make_float2(d2q[0], d2q[1]);
  st.last[lane] = make_uint2(last[0], last[1]);
  uint32_t npairs = 0;

  // Phases 1 and 3: this lane's entry of the group and row of the sub-block.
  const uint32_t e = lane & 7u, q = lane >> 3;
  const float px0 = (float)wk.bx + 0.5f;
  const f2 pyq = f2_make((float)(wk.by + q) + 0.5f, (float)(wk.by + q + 4u) + 0.5f);

  // Entries at or past every pixel's n_contrib contribute nothing: the tile's list is scanned from
  // its last contributor on, and the warp takes up the walk at its own (one that saturates early
  // beside one that doesn't has most of the list behind it).
  const uint32_t warp_last = __reduce_max_sync(0xffffffffu, max(last[0], last[1]));
  uint32_t min_last;  // over the image's pixels (the others are in no rectangle)
  {
    const uint32_t x = wk.bx + (lane & 7u), y = wk.by + (lane >> 3);
    min_last = x < wk.width && y < wk.height ? last[0] : 0xffffffffu;
    if (x < wk.width && y + 4u < wk.height) min_last = min(min_last, last[1]);
    min_last = __reduce_min_sync(0xffffffffu, min_last);
  }
  if (lane == 0) atomicMax(&tile_last, warp_last);
  wk.template barrier<Shape::kTiles>();
  const uint32_t n = tile_last;
  for (uint32_t first = 0; first < n; first += kListChunk) {
    if (first) wk.template barrier<Shape::kTiles>();
    const uint32_t total = min(n - first, (uint32_t)kListChunk);
    wk.scan(list, n - 1u - first, -1, total);
    wk.template barrier<Shape::kTiles>();
    Stager<typename W::Mask, kBwdStage> stager;
    const uint32_t past = n - min(n, first + warp_last);  // of this scan's entries, those past the warp's last
    stager.start(&list, past, total, wk.sub, st.queue);
    uint32_t buf = 0, next_g = 0, next_index = 0;
    uint32_t m = stager.fetch(rec, st.s[0][0], kBwdStage, &next_g, &next_index);
    while (m) {
      copy_async_wait();
      __syncwarp();
      const float4(*s)[kBwdStage] = st.s[buf];
      // Per staged entry (lane i: entry i): Gaussian, list position and the sub-block's columns
      // (bits 0-7) and rows (8-15) in its rectangle; bit 16 marks the scalar rule.
      const uint32_t cnt = m, stage_g = next_g, stage_place = n - 1u - first - next_index;
      uint32_t stage_mask = 0;
      if (lane < cnt) {
        const float4 r2 = s[2][lane];
        stage_mask = sub_block_mask(fbits(r2.z), fbits(r2.w), wk.bx, wk.by) |
                     (special_geometry(s[0][lane], s[1][lane]) ? 0x10000u : 0u);
      }
      buf ^= 1u;
      m = stager.fetch(rec, st.s[buf][0], kBwdStage, &next_g, &next_index);  // loads while these are walked
      for (uint32_t j0 = 0; j0 < cnt; j0 += kGroup) {
        // ---- Phase 1
        const uint32_t j = min(j0 + e, cnt - 1u);
        const bool valid = j0 + e < cnt;
        const float4 r0 = s[0][j], r1 = s[1][j];
        const float2 gb = *reinterpret_cast<const float2*>(&s[2][j]);
        const uint32_t gi = __shfl_sync(0xffffffffu, stage_g, j);
        const uint32_t place = __shfl_sync(0xffffffffu, stage_place, j);
        const uint32_t mask0 = __shfl_sync(0xffffffffu, stage_mask, j), mask = valid ? mask0 : 0u;
        const float A = r0.z, B = r0.w, opacity = r1.y, sigma_max = r1.z, sure = sigma_max - kSigmaEdge;
        const f2 dy = f2_sub(pyq, f2_splat(r0.y));
        const f2 cdy = f2_mul(f2_splat(r1.x), dy);
        // A row outside the rectangle gets sigma = inf.
        const float inf = __int_as_float(0x7f800000);
        f2 cdyy;
        {
          float lo, hi;
          f2_split(f2_mul(cdy, dy), lo, hi);
          cdyy = f2_make((mask >> (8u + q)) & 1u ? lo : inf, (mask >> (12u + q)) & 1u ? hi : inf);
        }
        uint32_t nearest = 0xffffffffu;  // bits of the smallest positive sigma - sure
        f2 sum = f2_splat(0.0f);         // of gauss: positive when a pixel takes the entry
        // sigma in [0, sure] as one unsigned comparison of the bits: sigma is never -0 (no product
        // or sum above gives it) and a negative or NaN sigma compares above. sure < 0 takes the
        // scalar rule.
        const uint32_t sure_bits = fbits(sure);
        const bool ordered = place < min_last;  // every pixel's n_contrib is past this entry
        if (__all_sync(0xffffffffu, ordered || !valid)) {
          evaluate_row<kCount, false>(st, e, q, px0, r0, dy, cdyy, mask, place, sure, sure_bits, nearest, sum, npairs);
        } else {
          evaluate_row<kCount, true>(st, e, q, px0, r0, dy, cdyy, mask, place, sure, sure_bits, nearest, sum, npairs);
        }
        bool any;
        {
          float lo, hi;
          f2_split(sum, lo, hi);
          any = lo > 0.0f || hi > 0.0f;
        }
        // Rare: a pixel within kSigmaEdge of sigma_max takes the correctly rounded exp for its
        // alpha test, and so do all pixels of an entry whose sigma may not be finite.
        const bool edge = valid && ((mask & 0x10000u) || nearest <= fbits(2.0f * kSigmaEdge));
        if (__any_sync(0xffffffffu, edge)) {
          if (edge) {
            any = false;
            for (uint32_t k = 0; k < 16; k++) {
              const uint32_t c = k >> 1, hi = k & 1u;
              const float dx = (px0 + (float)c) - r0.x, dyk = (float)(wk.by + q + 4u * hi) + 0.5f - r0.y;
              const float sg = 0.5f * (A * dx * dx + r1.x * dyk * dyk) + B * dx * dyk;
              const uint2 lp = st.last[8u * q + c];
              const bool in = ((mask >> c) & 1u) && ((mask >> (8u + q + 4u * hi)) & 1u) && place < (hi ? lp.y : lp.x);
              bool v = in && !(sg < 0.0f) && !(sg > sigma_max);
              if (v && !(sg <= sure)) v = !(opacity * crm::expf_cr(-sg) < SPLAT_ALPHA_MIN);
              any = any || v;
              reinterpret_cast<float*>(&st.h[e][8u * q + c])[hi] = v ? fast_exp(-sg) : 0.0f;
            }
          }
        }
        // Products within a relative band of the clamp are decided with the correctly rounded
        // exp (opacity below 0.99 never clamps).
        const bool clamps = !(opacity < SPLAT_ALPHA_MAX);
        if (__any_sync(0xffffffffu, clamps && any)) {
          if (clamps && any) {
            for (uint32_t k = 0; k < 16; k++) {
              const uint32_t c = k >> 1, hi = k & 1u;
              float* g = reinterpret_cast<float*>(&st.h[e][8u * q + c]) + hi;
              if (!(fabsf(opacity * *g - SPLAT_ALPHA_MAX) < SPLAT_ALPHA_MAX * kExpBand)) continue;
              const float dx = (px0 + (float)c) - r0.x, dyk = (float)(wk.by + q + 4u * hi) + 0.5f - r0.y;
              *g = crm::expf_cr(-(0.5f * (A * dx * dx + r1.x * dyk * dyk) + B * dx * dyk));
            }
          }
        }
        uint32_t taken = __ballot_sync(0xffffffffu, any);
        taken |= taken >> 16;
        taken = (taken | (taken >> 8)) & 0xffu;
        if (!taken) continue;
        const bool clamping = __any_sync(0xffffffffu, clamps);
        if (q == 0)
          st.color[e] = (taken >> e) & 1u ? make_float4(opacity, r1.w, gb.x, gb.y) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        __syncwarp();
        // ---- Phase 2
        if (clamping)
          walk_entries<true>(st, lane, pp);
        else
          walk_entries<false>(st, lane, pp);
        __syncwarp();
        // ---- Phase 3
        const f2 bdy = f2_mul(f2_splat(B), dy);
        f2 h0 = f2_splat(0.0f), h1 = h0, h2 = h0, gx = h0, gy = h0, w0 = h0, wr = h0, wg = h0, wb = h0;
        float ax = 0.0f, ay = 0.0f;
        f2 dx = f2_splat(px0 - r0.x);
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const float2 hv = st.h[e][8u * q + c], wv = st.w[e][8u * q + c];
          const float4 d01 = st.d01[8u * q + c];
          const float2 d2 = st.d2[8u * q + c];
          const f2 h = f2_make(hv.x, hv.y), w = f2_make(wv.x, wv.y);
          const f2 hx = f2_mul(h, dx);
          h0 = f2_add(h0, h);
          h1 = f2_add(h1, hx);
          h2 = f2_fma(hx, dx, h2);
          w0 = f2_add(w0, w);
          wr = f2_fma(w, f2_make(d01.x, d01.y), wr);
          wg = f2_fma(w, f2_make(d01.z, d01.w), wg);
          wb = f2_fma(w, f2_make(d2.x, d2.y), wb);
          const f2 hmx = f2_mul(h, f2_fma(f2_splat(A), dx, bdy)), hmy = f2_mul(h, f2_fma(f2_splat(B), dx, cdy));
          gx = f2_add(gx, hmx);
          gy = f2_add(gy, hmy);
          float lo, hi;
          f2_split(hmx, lo, hi);
          ax += fabsf(lo);
          ax += fabsf(hi);
          f2_split(hmy, lo, hi);
          ay += fabsf(lo);
          ay += fabsf(hi);
          dx = f2_add(dx, f2_splat(1.0f));
        }
        // Slots 0-11: d mean2d.x, .y, d conic A, B, C, d opacity, d r, g, b, |d mean2d.x|, |.y|,
        // sum(alpha T).
        float v[kSlots], lo, hi, dy0, dy1;
        f2_split(dy, dy0, dy1);
        f2_split(h0, lo, hi);
        const float syy = __fmaf_rn(dy1 * dy1, hi, (dy0 * dy0) * lo);
        v[5] = lo + hi;
        f2_split(h1, lo, hi);
        const float sxy = __fmaf_rn(dy1, hi, dy0 * lo);
        f2_split(h2, lo, hi);
        const float sxx = lo + hi;
        f2_split(gx, lo, hi);
        v[0] = opacity * (lo + hi);
        f2_split(gy, lo, hi);
        v[1] = opacity * (lo + hi);
        v[2] = -0.5f * opacity * sxx;
        v[3] = -opacity * sxy;
        v[4] = -0.5f * opacity * syy;
        f2_split(wr, lo, hi);
        v[6] = lo + hi;
        f2_split(wg, lo, hi);
        v[7] = lo + hi;
        f2_split(wb, lo, hi);
        v[8] = lo + hi;
        v[9] = fabsf(opacity) * ax;
        v[10] = fabsf(opacity) * ay;
        f2_split(w0, lo, hi);
        v[11] = lo + hi;
        // Two exchange stages over the entry's four lanes: 6 + 3 shuffles leave lane (e, q) with
        // slots 3 q .. 3 q + 2 (q's bit 1 chooses the half, bit 0 the half of the half).
        const bool b1 = lane & 16u, b0 = lane & 8u;
        float x6[6], x3[3];
#pragma unroll
        for (int i = 0; i < 6; i++)
          x6[i] = (b1 ? v[i + 6] : v[i]) + __shfl_xor_sync(0xffffffffu, b1 ? v[i] : v[i + 6], 16);
#pragma unroll
        for (int i = 0; i < 3; i++)
          x3[i] = (b0 ? x6[i + 3] : x6[i]) + __shfl_xor_sync(0xffffffffu, b0 ? x6[i] : x6[i + 3], 8);
        __syncwarp();  // every lane has read the rows: the first ones take the sums
        float* out = reinterpret_cast<float*>(st.w);
#pragma unroll
        for (int i = 0; i < 3; i++) out[e * kSlots + 3u * q + i] = x3[i];
        __syncwarp();
        const uint32_t i = lane / 3u, p = lane - 3u * i;  // lane 3 i + p: plane p of entry i
        const uint32_t target = __shfl_sync(0xffffffffu, gi, i & 7u);
        if (i < (uint32_t)kGroup && ((taken >> i) & 1u)) {
          const float4 t = reinterpret_cast<const float4*>(st.w)[lane];
          if (t.x != 0.0f || t.y != 0.0f || t.z != 0.0f || t.w != 0.0f) atomicAdd(&pgrad[p * (size_t)cap + target], t);
        }
        __syncwarp();
      }
    }
  }
  if (kCount) {
    unsigned long long np = npairs;
    for (int o = 16; o > 0; o >>= 1) np += __shfl_xor_sync(0xffffffffu, np, o);
    if (lane == 0 && np) atomicAdd(pairs, np);
  }
}

// ---------------------------------------------------------------------------------------
// Deterministic backward (16x16 tiles): the reference's own reduction, bit for bit.
//
// backward_tile (rasterize.rs:394-454) sums each entry's 11 slots over the pixels of its
// rectangle in row-major order, in unfused f32 arithmetic, and stores them per entry;
// rasterize_backward (:480-503) then sums every Gaussian's entries in entry order. Here a
// block walks its tile's list in reverse like the atomic kernel, but every pixel writes its
// per-entry contribution to shared memory (kDetGroup entries at a time) and one thread per
// (entry, slot) adds the contributions of the rectangle's pixels in row-major order; the
// per-entry sums go to a slot array indexed by the entry's emission index (Gaussian-major,
// rasterize.rs:76-97), which entry_slots_reduce_kernel sums per Gaussian. Pixels that do not
// contribute add +0.0, which leaves a sum unchanged (a sum that starts at +0.0 is never -0.0),
// so the totals equal the reference's, which skips them. The arithmetic per pixel is the
// reference's operation for operation: the correctly rounded exp of the forward, true
// divisions, no contraction (the file is compiled with --fmad=false), and dalpha built from
// 0.0 as the reference builds it.
// ---------------------------------------------------------------------------------------
constexpr int kDetGroup = 8;
constexpr int kDetChunk = 64;
constexpr size_t kDetSmemBytes = (size_t)kDetGroup * kSlots * 256 * sizeof(float);

// Emission index of the entry of Gaussian g in tile (tx, ty): its entries are emitted row by
// row over its tile rectangle (rasterize.rs:87-96).
__device__ __forceinline__ uint32_t entry_index(const float4* __restrict__ rec,
                                                const uint32_t* __restrict__ entry_offset, uint32_t g, uint32_t tx,
                                                uint32_t ty) {
  const float4 r3 = rec[4 * (size_t)g + 3];
  const uint32_t tmin = fbits(r3.z), tmax = fbits(r3.w);
  const uint32_t tx0 = tmin & 0xffffu, ty0 = tmin >> 16, w = (tmax & 0xffffu) - tx0;
  return entry_offset[g] + (ty - ty0) * w + (tx - tx0);
}

__global__ void __launch_bounds__(256) raster_bwd_det_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ gauss, const uint2* __restrict__ ranges,
    const uint32_t* __restrict__ entry_offset, int64_t e_cap, uint32_t width, uint32_t height, uint32_t tiles_x,
    float bg0, float bg1, float bg2, const float* __restrict__ final_t, const uint32_t* __restrict__ n_contrib,
    const float* __restrict__ dimage, float* __restrict__ eslot) {
  extern __shared__ float cbuf[];  // [kDetGroup][kSlots][256], pixel index row-major in the tile
  __shared__ float4 s0[kDetChunk], s1[kDetChunk];
  __shared__ float2 s2[kDetChunk];
  __shared__ uint32_t srect[kDetChunk];
  __shared__ uint32_t sent[kDetChunk];
  __shared__ uint32_t s_max_last;
  const uint32_t tile = blockIdx.x;
  const uint32_t tx = tile % tiles_x, ty = tile / tiles_x;
  const uint32_t ox = tx * 16u, oy = ty * 16u;
  const uint32_t lx = threadIdx.x & 15u, ly = threadIdx.x >> 4;
  const uint32_t x = ox + lx, y = oy + ly;
  const bool inside = x < width && y < height;
  const float px = (float)x + 0.5f, py = (float)y + 0.5f;
  const uint2 range = ranges[tile];
  const uint32_t list_len = range.y - range.x;
  // Clipped extent of the tile (tile_geom, rasterize.rs:203-215).
  const uint32_t gw = min(width - ox, 16u), gh = min(height - oy, 16u);

  uint32_t last = 0;
  float T = 1.0f, t_fin = 1.0f, d0 = 0.0f, d1 = 0.0f, d2 = 0.0f, bg_dot = 0.0f;
  if (inside) {
    const size_t pix = (size_t)y * width + x;
    last = min(n_contrib[pix], list_len);
    T = final_t[pix];
    t_fin = T;
    d0 = dimage[3 * pix];
    d1 = dimage[3 * pix + 1];
    d2 = dimage[3 * pix + 2];
    bg_dot = bg0 * d0 + bg1 * d1 + bg2 * d2;
  }
  float acc_r = 0.0f, acc_g = 0.0f, acc_b = 0.0f, last_alpha = 0.0f, lc_r = 0.0f, lc_g = 0.0f, lc_b = 0.0f;
  if (threadIdx.x == 0) s_max_last = 0;
  __syncthreads();
  const uint32_t wmax = __reduce_max_sync(0xffffffffu, last);
  if ((threadIdx.x & 31u) == 0) atomicMax(&s_max_last, wmax);
  __syncthreads();
  const uint32_t max_last = s_max_last;
  // Entries no pixel reaches keep zero slots.
  for (uint32_t k = max_last + threadIdx.x; k < list_len; k += 256) {
    const uint32_t e = entry_index(rec, entry_offset, gauss[range.x + k], tx, ty);
    if (e < e_cap) {
#pragma unroll
      for (int q = 0; q < kSlots; q++) eslot[(size_t)e * kSlots + q] = 0.0f;
    }
  }

  for (uint32_t cend = max_last; cend > 0;) {
    const uint32_t cstart = cend > (uint32_t)kDetChunk ? cend - kDetChunk : 0u;
    const uint32_t cnt = cend - cstart;
    for (uint32_t e = threadIdx.x; e < cnt; e += 256) {
      const uint32_t g = gauss[range.x + cstart + e];
      s0[e] = rec[4 * (size_t)g];
      s1[e] = rec[4 * (size_t)g + 1];
      const float4 e2 = rec[4 * (size_t)g + 2];
      s2[e] = make_float2(e2.x, e2.y);
      srect[e] = tile_rect_masks<16, 16>(fbits(e2.z), fbits(e2.w), ox, oy);
      sent[e] = entry_index(rec, entry_offset, g, tx, ty);
    }
    __syncthreads();
    for (uint32_t gend = cnt; gend > 0;) {
      const uint32_t gstart = gend > (uint32_t)kDetGroup ? gend - kDetGroup : 0u;
      // Each pixel's contributions to the group's entries, in reverse depth order.
      for (uint32_t kk = gend; kk-- > gstart;) {
        const uint32_t j = gend - 1u - kk;
        const uint32_t rm = srect[kk];
        if (!inside || !((rm >> lx) & 1u) || !((rm >> (16u + ly)) & 1u)) continue;  // outside the rectangle
        float c[kSlots];
#pragma unroll
        for (int q = 0; q < kSlots; q++) c[q] = 0.0f;
        const uint32_t k = cstart + kk;
        const float4 e0 = s0[kk], e1 = s1[kk];
        const float2 e2 = s2[kk];
        float gval, alpha;
        if (k < last && evaluate_ref(px, py, e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, &gval, &alpha)) {
          const float col_r = e1.w, col_g = e2.x, col_b = e2.y;
          T = T / (1.0f - alpha);
          const float t = T;
          float dalpha = 0.0f;
          acc_r = last_alpha * lc_r + (1.0f - last_alpha) * acc_r;
          dalpha += (col_r - acc_r) * d0;
          c[6] = alpha * t * d0;
          acc_g = last_alpha * lc_g + (1.0f - last_alpha) * acc_g;
          dalpha += (col_g - acc_g) * d1;
          c[7] = alpha * t * d1;
          acc_b = last_alpha * lc_b + (1.0f - last_alpha) * acc_b;
          dalpha += (col_b - acc_b) * d2;
          c[8] = alpha * t * d2;
          dalpha *= t;
          lc_r = col_r;
          lc_g = col_g;
          lc_b = col_b;
          last_alpha = alpha;
          dalpha += -t_fin / (1.0f - alpha) * bg_dot;
          c[11] = alpha * t;
          const float opacity = e1.y;
          if (opacity * gval < SPLAT_ALPHA_MAX) {
            c[5] = gval * dalpha;
            const float dgauss = opacity * dalpha;
            const float dsigma = -dgauss * gval;
            const float dx = px - e0.x;
            const float dy = py - e0.y;
            const float ddx = dsigma * (e0.z * dx + e0.w * dy);
            const float ddy = dsigma * (e0.w * dx + e1.x * dy);
            c[0] = -ddx;
            c[1] = -ddy;
            c[2] = dsigma * 0.5f * dx * dx;
            c[3] = dsigma * dx * dy;
            c[4] = dsigma * 0.5f * dy * dy;
            c[9] = fabsf(ddx);
            c[10] = fabsf(ddy);
          }
        }
#pragma unroll
        for (int q = 0; q < kSlots; q++) cbuf[((size_t)j * kSlots + q) * 256 + threadIdx.x] = c[q];
      }
      __syncthreads();
      // One thread per (entry, slot): the rectangle's pixels in row-major order.
      if (threadIdx.x < (gend - gstart) * (uint32_t)kSlots) {
        const uint32_t j = threadIdx.x / kSlots, q = threadIdx.x % kSlots;
        const uint32_t kk = gend - 1u - j;
        const uint32_t rm = srect[kk];
        const uint32_t cols = rm & 0xffffu, rows = rm >> 16;
        float a = 0.0f;
        if (cols && rows) {
          const uint32_t x0 = __ffs(cols) - 1u, x1 = min(32u - __clz(cols), gw);
          const uint32_t y0 = __ffs(rows) - 1u, y1 = min(32u - __clz(rows), gh);
          const float* b = cbuf + ((size_t)j * kSlots + q) * 256;
          for (uint32_t yy = y0; yy < y1; yy++)
            for (uint32_t xx = x0; xx < x1; xx++) a += b[yy * 16u + xx];
        }
        const uint32_t e = sent[kk];
        if (e < e_cap) eslot[(size_t)e * kSlots + q] = a;
      }
      __syncthreads();
      gend = gstart;
    }
    cend = cstart;
  }
}

// The per-Gaussian sum of rasterize_backward (rasterize.rs:480-503): entries in emission
// order from 0.0, into the screen-space gradient planes (written, not accumulated).
__global__ void __launch_bounds__(256) entry_slots_reduce_kernel(const uint32_t* __restrict__ entry_offset,
                                                                 int64_t n, const float4* __restrict__ eslot,
                                                                 int64_t e_cap, float4* __restrict__ pgrad,
                                                                 int64_t cap) {
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const int64_t s = entry_offset[g], e = min((int64_t)entry_offset[g + 1], e_cap);
  float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a, c = a;
  for (int64_t i = s; i < e; i++) {
    const float4 u = eslot[3 * i], v = eslot[3 * i + 1], w = eslot[3 * i + 2];
    a.x += u.x; a.y += u.y; a.z += u.z; a.w += u.w;
    b.x += v.x; b.y += v.y; b.z += v.z; b.w += v.w;
    c.x += w.x; c.y += w.y; c.z += w.z; c.w += w.w;
  }
  pgrad[g] = a;
  pgrad[cap + g] = b;
  pgrad[2 * cap + g] = c;
}

Status launch_raster_bwd_det(Ctx* c, const float* proj, const uint32_t* gauss, const uint32_t* ranges,
                             const uint32_t* entry_offset, int64_t n, int64_t e_cap, uint32_t width, uint32_t height,
                             const float bg[3], const float* final_t, const uint32_t* n_contrib, const float* dimage,
                             float* eslot, float* pgrad, int64_t cap) {
  if (!c->raster.reference_tiles())
    return Status::make(SPLAT_ERR_INVALID, "the deterministic backward needs the reference's 16x16 tiles");
  static bool attr_set[64] = {};
  if (c->device >= 0 && c->device < 64 && !attr_set[c->device]) {
    SPLAT_CUDA(cudaFuncSetAttribute(raster_bwd_det_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kDetSmemBytes));
    attr_set[c->device] = true;
  }
  const uint32_t tiles_x = c->raster.tiles_x(width);
  const uint32_t blocks = c->raster.tiles(width, height);
  if (blocks > 0 && e_cap > 0) {
    raster_bwd_det_kernel<<<blocks, 256, kDetSmemBytes, c->stream>>>(
        reinterpret_cast<const float4*>(proj), gauss, reinterpret_cast<const uint2*>(ranges), entry_offset, e_cap,
        width, height, tiles_x, bg[0], bg[1], bg[2], final_t, n_contrib, dimage, eslot);
    c->launches.count++;
    SPLAT_LAUNCHED("raster_bwd_det_kernel");
  }
  if (n > 0) {
    entry_slots_reduce_kernel<<<ceil_div(n, 256), 256, 0, c->stream>>>(
        entry_offset, n, reinterpret_cast<const float4*>(eslot), e_cap, reinterpret_cast<float4*>(pgrad), cap);
    c->launches.count++;
    SPLAT_LAUNCHED("entry_slots_reduce_kernel");
  }
  return Status::ok();
}

// Expands CALL(TW, TH, CH) for the configuration rc; an unsupported one is an error.
#define SPLAT_RASTER_DISPATCH(rc, CALL)                                                       \
  do {                                                                                         \
    const uint32_t w_ = (rc).tile_w, h_ = (rc).tile_h, c_ = (rc).chunk;                        \
    if (w_ == 16 && h_ == 16 && c_ == 256) CALL(16, 16, 256);                                  \
    else if (w_ == 16 && h_ == 16 && c_ == 128) CALL(16, 16, 128);                             \
    else if (w_ == 16 && h_ == 16 && c_ == 64) CALL(16, 16, 64);                               \
    else if (w_ == 16 && h_ == 16 && c_ == 32) CALL(16, 16, 32);                               \
    else if (w_ == 8 && h_ == 8 && c_ == 256) CALL(8, 8, 256);                                 \
    else if (w_ == 8 && h_ == 8 && c_ == 128) CALL(8, 8, 128);                                 \
    else if (w_ == 8 && h_ == 8 && c_ == 64) CALL(8, 8, 64);                                   \
    else if (w_ == 8 && h_ == 8 && c_ == 32) CALL(8, 8, 32);                                   \
    else if (w_ == 16 && h_ == 32 && c_ == 256) CALL(16, 32, 256);                             \
    else if (w_ == 16 && h_ == 32 && c_ == 128) CALL(16, 32, 128);                             \
    else if (w_ == 16 && h_ == 32 && c_ == 64) CALL(16, 32, 64);                               \
    else if (w_ == 16 && h_ == 32 && c_ == 32) CALL(16, 32, 32);                               \
    else return Status::make(SPLAT_ERR_INVALID, "unsupported raster configuration");           \
  } while (0)

// Launches a walking kernel over `tiles` tiles. Its shared memory is above the default limit,
// which is raised on the kernel's first use on a device.
template <typename Shape, typename Smem, typename... P, typename... A>
static Status launch_walk(Ctx* c, void (*kernel)(P...), uint32_t tiles, A... args) {
  static std::mutex guard;
  static std::set<std::pair<int, const void*>> ready;
  {
    std::lock_guard<std::mutex> lock(guard);
    const std::pair<int, const void*> key(c->device, reinterpret_cast<const void*>(kernel));
    if (!ready.count(key)) {
      SPLAT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Smem)));
      ready.insert(key);
    }
  }
  return launch_chained(c, "compositing kernel", kernel, ceil_div(tiles, Shape::kTiles), 32 * Shape::kWarps,
                        sizeof(Smem), args...);
}

Status launch_raster_fwd(Ctx* c, const float* proj, const uint32_t* gauss, const uint32_t* ranges, uint32_t width,
                         uint32_t height, const float bg[3], float* image, float* final_t, uint32_t* n_contrib,
                         uint64_t* pairs, const BatchTable* bt, uint32_t tiles_cap) {
  const RasterConfig& rc = c->raster;
  const uint32_t tiles_x = rc.tiles_x(width);
  const uint32_t tiles = bt ? tiles_cap : rc.tiles(width, height);
  if (tiles == 0) return Status::ok();
#define SPLAT_FWDK(TW, TH, K)                                                                                     \
  SPLAT_TRY((launch_walk<FwdShape<TW, TH>, FwdSmem<TW, TH>>(                                                     \
      c, raster_fwd_kernel<TW, TH, K>, tiles, reinterpret_cast<const float4*>(proj), gauss,                      \
      reinterpret_cast<const uint2*>(ranges), tiles, width, height, tiles_x, bg[0], bg[1], bg[2], image, final_t, \
      n_contrib, reinterpret_cast<unsigned long long*>(pairs), bt)))
#define SPLAT_FWD(TW, TH) \
  if (pairs) SPLAT_FWDK(TW, TH, true); else SPLAT_FWDK(TW, TH, false)
  if (rc.tile_w == 16 && rc.tile_h == 16) {
    SPLAT_FWD(16, 16);
  } else if (rc.tile_w == 16 && rc.tile_h == 32) {
    SPLAT_FWD(16, 32);
  } else if (rc.tile_w == 8 && rc.tile_h == 8) {
    SPLAT_FWD(8, 8);
  } else {
    return Status::make(SPLAT_ERR_INVALID, "unsupported raster configuration");
  }
#undef SPLAT_FWD
#undef SPLAT_FWDK
  return Status::ok();
}

Status launch_raster_bwd(Ctx* c, const float* proj, const uint32_t* gauss, const uint32_t* ranges, uint32_t width,
                         uint32_t height, const float bg[3], const float* final_t, const uint32_t* n_contrib,
                         const float* dimage, float* pgrad, int64_t cap, uint64_t* pairs, const BatchTable* bt,
                         uint32_t tiles_cap) {
  const RasterConfig& rc = c->raster;
  const uint32_t tiles_x = rc.tiles_x(width);
  const uint32_t blocks = bt ? tiles_cap : rc.tiles(width, height);
  if (blocks == 0) return Status::ok();
#define SPLAT_BWD(TW, TH, CH, P)                                                                                  \
  SPLAT_TRY(launch_chained(c, "raster_bwd_kernel", raster_bwd_kernel<TW, TH, CH, P>, blocks, TW * TH / P, 0, \
      reinterpret_cast<const float4*>(proj), gauss, reinterpret_cast<const uint2*>(ranges), width, height, tiles_x, \
      bg[0], bg[1], bg[2], final_t, n_contrib, dimage, reinterpret_cast<float4*>(pgrad), cap,                     \
      reinterpret_cast<unsigned long long*>(pairs), bt))
#define SPLAT_BWD1(TW, TH, CH) SPLAT_BWD(TW, TH, CH, 1)
#define SPLAT_BWD2X(TW, TH, K, R)                                                                                   \
  SPLAT_TRY((launch_walk<BwdShape<TW, TH>, BwdSmem<TW, TH>>(                                                     \
      c, raster_bwd_x2_kernel<TW, TH, K, R>, blocks, reinterpret_cast<const float4*>(proj), gauss,                  \
      reinterpret_cast<const uint2*>(ranges), blocks, width, height, tiles_x, bg[0], bg[1], bg[2], final_t,      \
      n_contrib, dimage, reinterpret_cast<float4*>(pgrad), cap, reinterpret_cast<unsigned long long*>(pairs), bt)))
// 16 warps per SM in up to 128 registers, or, for views of many 16x16 tiles, 20 warps in 96. The
// line lies at 16 tiles per SM (2,368): 16 against 20 warps 22.9 / 24.0 us at 128x96 (2k Gaussians),
// 78.8 / 83.5 at 256x256 (34k), 84.4 / 90.2 at 640x480 (34k, 1,200 tiles), 53.5 / 54.4 at 800x600
// (100k, 1,900 tiles); 65.1 / 62.5 at 1280x720 (100k, 3,600 tiles), 256 / 256 at 1297x840 (187k),
// 674 / 666 at 1920x1080 (1M). 8x8 tiles spill at 20 warps and are 8-25% slower at every size
// (668 / 737 us in the last); a 16x32 block has eight warps, so two blocks per SM either way.
#define SPLAT_BWD2(TW, TH)                                                                                   \
  constexpr int kMany = TW == 16 && TH == 16 ? 20 : 16;                                                      \
  if (pairs) SPLAT_BWD2X(TW, TH, true, 16); else if (blocks <= 16u * (uint32_t)c->sm_count)                  \
    SPLAT_BWD2X(TW, TH, false, 16); else SPLAT_BWD2X(TW, TH, false, kMany)
  if (rc.ppl == 2) {
    if (rc.tile_w == 16 && rc.tile_h == 16) {
      SPLAT_BWD2(16, 16);
    } else if (rc.tile_w == 16 && rc.tile_h == 32) {
      SPLAT_BWD2(16, 32);
    } else if (rc.tile_w == 8 && rc.tile_h == 8) {
      SPLAT_BWD2(8, 8);
    } else {
      return Status::make(SPLAT_ERR_INVALID, "unsupported raster configuration");
    }
    return Status::ok();
  }
  SPLAT_RASTER_DISPATCH(rc, SPLAT_BWD1);
#undef SPLAT_BWD2
#undef SPLAT_BWD2X
#undef SPLAT_BWD1
#undef SPLAT_BWD
  return Status::ok();
}

}  // namespace splat
