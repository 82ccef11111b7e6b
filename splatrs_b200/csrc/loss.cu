// Photometric loss (1 - lambda) L1 + lambda (1 - SSIM) with its gradient (reference
// src/loss.rs:14-190), as two tiled kernels.
//
//   ssim_fwd: per output tile and channel, the 11-tap separable zero-padded blur of x, y, x^2,
//     y^2 and xy from a shared-memory tile with a 5-pixel halo; per-pixel SSIM and its partial
//     derivatives w.r.t. mu_x, E[x^2], E[xy] (written to scratch); the block's sums of SSIM,
//     |x - y| and the clamped squared error for PSNR (loss.rs:175-190).
//   ssim_bwd: the same blur of the three partial maps (the blur is self-adjoint,
//     loss.rs:124-127) and the gradient of the whole loss w.r.t. the prediction; its first block
//     adds up the blocks' sums.
// The target can be the view's 8-bit pixels, converted exactly as View::to_real does
// (reference src/dataset.rs:23-25), or floats. Blur sums run over the window in the
// reference's order, so the blurred maps, the partial maps and the gradient are bit-identical
// to the reference's; only the three scalar sums depend on summation order (accumulated in
// double here). Blurs of two maps run together as f32x2 pairs (pair.cuh: each half rounded as
// the scalar operation), so a tap of (x, y) or of (x^2, y^2) is one paired multiply and one
// paired add.
#include "common.cuh"
#include "kernels.cuh"
#include "pair.cuh"

namespace splat {

constexpr int kHalo = 5;  // SSIM_WINDOW / 2

struct LossKernel {
  float w[6];  // the window's weights are symmetric: w[|k - 5|] is tap k's
};
__host__ __device__ constexpr int tap_weight(int k) { return k < 5 ? 5 - k : k - 5; }

// View::to_real of an 8-bit value (reference src/dataset.rs:23-25): v / 255 rounded once. The
// quotient estimate is corrected by its exact remainder; equal to the division for all 256
// values (checked on the host).
__device__ __forceinline__ float u8_to_real(uint8_t v) {
  const float x = (float)v, r = 1.0f / 255.0f, q = x * r;
  return __fmaf_rn(__fmaf_rn(-255.0f, q, x), r, q);
}
__device__ __forceinline__ float load_target(const void* target, int target_u8, size_t idx) {
  if (target_u8) return u8_to_real(static_cast<const uint8_t*>(target)[idx]);
  return static_cast<const float*>(target)[idx];
}

// Loss, mean SSIM and PSNR of a view from its blocks' sums (loss.rs:147-154, :175-190), added by
// one block in block order: out = ((1 - lambda) l1 + lambda (1 - ssim), ssim, psnr).
template <int THREADS>
__device__ __forceinline__ void finalize_loss(const double* __restrict__ partial, uint32_t count, uint64_t n,
                                              float lambda, double (*red)[THREADS / 32], float* __restrict__ out) {
  double s[3] = {0.0, 0.0, 0.0};
  for (uint32_t k = threadIdx.x; k < count; k += THREADS)
#pragma unroll
    for (int q = 0; q < 3; q++) s[q] += partial[3 * (size_t)k + q];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
    if ((threadIdx.x & 31) == 0) red[q][threadIdx.x >> 5] = s[q];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int q = 0; q < 3; q++) {
      s[q] = 0.0;
      for (int w = 0; w < THREADS / 32; w++) s[q] += red[q][w];
    }
    const float inv_n = 1.0f / (float)n;
    const float l1 = (float)s[1] * inv_n;
    const float ssim = (float)(s[0] / (double)n);
    out[0] = (1.0f - lambda) * l1 + lambda * (1.0f - ssim);
    out[1] = ssim;
    const double mse = s[2] / (double)(n > 0 ? n : 1);
    out[2] = mse <= 0.0 ? INFINITY : (float)(-10.0 * log10(mse));
  }
  __syncthreads();
}

// ---------------------------------------------------------------------------------------
// Large views: a block takes all channels of a 32 x 32 tile in turn, two outputs per thread. The
// blocks' sums go to slots that the backward's first block adds up (no launch to clear, no launch
// to finish): 1297x840 120 -> 108 us, 1920x1080 206 -> 192 us for the whole loss. Tiles of 64 rows
// with eight outputs per thread and one channel per block were slower here (121 and 248 us: every
// channel's block reads the interleaved pixels again).
// ---------------------------------------------------------------------------------------
constexpr int kLT = kLossTile;     // output tile edge
constexpr int kLE = kLT + 2 * kHalo;
constexpr int kLossThreads = 256;
constexpr int kRB = 2;             // consecutive outputs per thread in each blur pass
static_assert(kLT % kRB == 0, "blocks of kRB outputs tile the output rows and columns");

// Sums: [0] SSIM, [1] |x - y|, [2] squared clamped error (PSNR), one triple per block.
__global__ void __launch_bounds__(kLossThreads) ssim_fwd_kernel(const float* __restrict__ pred,
                                                                const void* __restrict__ target_arg, int target_u8,
                                                                uint32_t width, uint32_t height, LossKernel K,
                                                                float* __restrict__ dmaps, double* __restrict__ sums,
                                                                const StepParams* __restrict__ sp,
                                                                const BatchTable* __restrict__ bt) {
  chain_begin();
  const void* target = sp ? sp->target : target_arg;
  int bxi = blockIdx.x, byi = blockIdx.y;
  if (bt) {  // a batch: flat block index -> view, block within the view, buffer offsets
    if (blockIdx.x >= bt->loss_start[bt->views]) return;
    const int v = batch_view_of(bt->loss_start, bt->views, blockIdx.x);
    const uint32_t local = blockIdx.x - bt->loss_start[v];
    bxi = local % bt->loss_blocks_x[v];
    byi = local / bt->loss_blocks_x[v];
    width = bt->cam[v].width;
    height = bt->cam[v].height;
    pred += 3 * bt->pix_start[v];
    target = bt->target[v];
    dmaps += 9 * bt->pix_start[v];
  }
  __shared__ float2 xy_tile[kLE][kLE];             // (prediction, target)
  __shared__ float2 h01[kLE][kLT], h23[kLE][kLT];  // horizontal blurs of (x, y) and (x^2, y^2)
  __shared__ float h4[kLE][kLT];                   // and of x y
  __shared__ double red[3][kLossThreads / 32];
  const int ox0 = bxi * kLT, oy0 = byi * kLT;
  const int tid = threadIdx.x;
  const float c1 = 0.01f * 0.01f, c2 = 0.03f * 0.03f;
  f2 wp[11];
#pragma unroll
  for (int k = 0; k < 11; k++) wp[k] = f2_splat(K.w[tap_weight(k)]);
  double s_ssim = 0.0, s_l1 = 0.0, s_se = 0.0;
  for (int ch = 0; ch < 3; ch++) {
    for (int i = tid; i < kLE * kLE; i += kLossThreads) {
      const int r = i / kLE, c = i % kLE;
      const int gy = oy0 - kHalo + r, gx = ox0 - kHalo + c;
      float vx = 0.0f, vy = 0.0f;
      if (gx >= 0 && gx < (int)width && gy >= 0 && gy < (int)height) {
        const size_t idx = ((size_t)gy * width + gx) * 3 + ch;
        vx = pred[idx];
        vy = load_target(target, target_u8, idx);
      }
      xy_tile[r][c] = make_float2(vx, vy);
    }
    __syncthreads();
    // Horizontal pass (loss.rs:42-56) for every halo row: a thread takes kRB consecutive
    // output columns of a row and streams their kRB + 10 inputs once, each tap added in
    // window order. Taps outside the image read the tile's zero padding and add +0.0,
    // which leaves every sum as the reference's (it skips them).
    for (int item = tid; item < kLE * (kLT / kRB); item += kLossThreads) {
      const int r = item / (kLT / kRB), c0 = (item % (kLT / kRB)) * kRB;
      f2 a01[kRB], a23[kRB];
      float a4[kRB];
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        a01[o] = a23[o] = f2_splat(0.0f);
        a4[o] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < kRB + 10; q++) {
        const float2 t = xy_tile[r][c0 + q];
        const f2 v = f2_make(t.x, t.y), sq = f2_mul(v, v);
        const float xy = t.x * t.y;
#pragma unroll
        for (int o = 0; o < kRB; o++) {
          const int k = q - o;
          if (k < 0 || k > 10) continue;
          a01[o] = f2_add(a01[o], f2_mul(wp[k], v));
          a23[o] = f2_add(a23[o], f2_mul(wp[k], sq));
          a4[o] += K.w[tap_weight(k)] * xy;
        }
      }
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        float lo, hi;
        f2_split(a01[o], lo, hi);
        h01[r][c0 + o] = make_float2(lo, hi);
        f2_split(a23[o], lo, hi);
        h23[r][c0 + o] = make_float2(lo, hi);
        h4[r][c0 + o] = a4[o];
      }
    }
    __syncthreads();
    // Vertical pass (loss.rs:58-70) and per-pixel SSIM (loss.rs:101-119): a thread takes kRB
    // consecutive rows of a column, streamed the same way.
    for (int item = tid; item < kLT * (kLT / kRB); item += kLossThreads) {
      const int c = item % kLT, r0 = (item / kLT) * kRB;
      f2 m01[kRB], e23[kRB];
      float exy_[kRB];
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        m01[o] = e23[o] = f2_splat(0.0f);
        exy_[o] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < kRB + 10; q++) {
        const float2 t01 = h01[r0 + q][c], t23 = h23[r0 + q][c];
        const float t4 = h4[r0 + q][c];
        const f2 v01 = f2_make(t01.x, t01.y), v23 = f2_make(t23.x, t23.y);
#pragma unroll
        for (int o = 0; o < kRB; o++) {
          const int k = q - o;
          if (k < 0 || k > 10) continue;
          m01[o] = f2_add(m01[o], f2_mul(wp[k], v01));
          e23[o] = f2_add(e23[o], f2_mul(wp[k], v23));
          exy_[o] += K.w[tap_weight(k)] * t4;
        }
      }
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        const int r = r0 + o;
        const int gy = oy0 + r, gx = ox0 + c;
        if (gx >= (int)width || gy >= (int)height) continue;
        float mx, my, exx, eyy;
        f2_split(m01[o], mx, my);
        f2_split(e23[o], exx, eyy);
        const float exy = exy_[o];
        const float sx2 = exx - mx * mx;
        const float sy2 = eyy - my * my;
        const float sxy = exy - mx * my;
        const float n1 = 2.0f * mx * my + c1;
        const float n2 = 2.0f * sxy + c2;
        const float d1 = mx * mx + my * my + c1;
        const float d2 = sx2 + sy2 + c2;
        const float num = n1 * n2;
        const float den = d1 * d2;
        const float sv = num / den;
        const float dn_dmx = 2.0f * my * n2 - 2.0f * my * n1;
        const float dd_dmx = 2.0f * mx * d2 - 2.0f * mx * d1;
        // The partial maps are planar (map, channel, pixel), so that the backward's per-channel
        // tile loads are contiguous.
        const size_t pix = (size_t)gy * width + gx, npix = (size_t)width * height;
        dmaps[(size_t)ch * npix + pix] = (dn_dmx * den - num * dd_dmx) / (den * den);
        dmaps[(size_t)(3 + ch) * npix + pix] = -num * d1 / (den * den);
        dmaps[(size_t)(6 + ch) * npix + pix] = 2.0f * n1 / den;
        const float2 xy = xy_tile[r + kHalo][c + kHalo];
        const float x = xy.x, y = xy.y;
        s_ssim += (double)sv;
        s_l1 += (double)fabsf(x - y);
        const double e = (double)fminf(fmaxf(x, 0.0f), 1.0f) - (double)fminf(fmaxf(y, 0.0f), 1.0f);
        s_se += e * e;
      }
    }
    __syncthreads();
  }
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s_ssim += __shfl_xor_sync(0xffffffffu, s_ssim, o);
    s_l1 += __shfl_xor_sync(0xffffffffu, s_l1, o);
    s_se += __shfl_xor_sync(0xffffffffu, s_se, o);
  }
  if (lane == 0) {
    red[0][warp] = s_ssim;
    red[1][warp] = s_l1;
    red[2][warp] = s_se;
  }
  __syncthreads();
  if (tid < 3) {
    double t = 0.0;
    for (int w = 0; w < kLossThreads / 32; w++) t += red[tid][w];
    sums[3 * ((size_t)blockIdx.y * gridDim.x + blockIdx.x) + tid] = t;
  }
}

// Gradient of the loss w.r.t. the prediction (loss.rs:124-133, :155-169); the first block also
// finishes the loss values.
__global__ void __launch_bounds__(kLossThreads) ssim_bwd_kernel(const float* __restrict__ pred,
                                                                const void* __restrict__ target_arg, int target_u8,
                                                                uint32_t width, uint32_t height, LossKernel K,
                                                                const float* __restrict__ dmaps,
                                                                const double* __restrict__ sums, float lambda,
                                                                float* __restrict__ grad, float* __restrict__ out3,
                                                                const StepParams* __restrict__ sp,
                                                                const BatchTable* __restrict__ bt) {
  chain_begin();
  __shared__ double red[3][kLossThreads / 32];
  if (blockIdx.x == 0 && blockIdx.y == 0) {
    if (bt) {
      for (int v = 0; v < bt->views; v++)
        finalize_loss<kLossThreads>(sums + 3 * (size_t)bt->loss_start[v], bt->loss_start[v + 1] - bt->loss_start[v],
                                    3 * (bt->pix_start[v + 1] - bt->pix_start[v]), lambda, red, out3 + 3 * v);
    } else {
      finalize_loss<kLossThreads>(sums, gridDim.x * gridDim.y, 3 * (uint64_t)width * height, lambda, red, out3);
    }
  }
  const void* target = sp ? sp->target : target_arg;
  int bxi = blockIdx.x, byi = blockIdx.y;
  float scale = 1.0f;  // a batch averages the views' gradients
  if (bt) {
    if (blockIdx.x >= bt->loss_start[bt->views]) return;
    const int v = batch_view_of(bt->loss_start, bt->views, blockIdx.x);
    const uint32_t local = blockIdx.x - bt->loss_start[v];
    bxi = local % bt->loss_blocks_x[v];
    byi = local / bt->loss_blocks_x[v];
    width = bt->cam[v].width;
    height = bt->cam[v].height;
    pred += 3 * bt->pix_start[v];
    target = bt->target[v];
    dmaps += 9 * bt->pix_start[v];
    grad += 3 * bt->pix_start[v];
    scale = bt->inv_views;
  }
  __shared__ float2 sm01[kLE][kLE];  // partial maps w.r.t. mu_x and E[x^2]
  __shared__ float sm2[kLE][kLE];    // and w.r.t. E[xy]
  __shared__ float2 h01[kLE][kLT];
  __shared__ float h2[kLE][kLT];
  const int ox0 = bxi * kLT, oy0 = byi * kLT;
  const int tid = threadIdx.x;
  const size_t npix3 = (size_t)width * height * 3;
  const float inv_n = 1.0f / (float)npix3;
  const float w1 = (1.0f - lambda) * inv_n;
  f2 wp[11];
#pragma unroll
  for (int k = 0; k < 11; k++) wp[k] = f2_splat(K.w[tap_weight(k)]);
  for (int ch = 0; ch < 3; ch++) {
    for (int i = tid; i < kLE * kLE; i += kLossThreads) {
      const int r = i / kLE, c = i % kLE;
      const int gy = oy0 - kHalo + r, gx = ox0 - kHalo + c;
      float a = 0.0f, b = 0.0f, e = 0.0f;
      if (gx >= 0 && gx < (int)width && gy >= 0 && gy < (int)height) {
        const size_t pix = (size_t)gy * width + gx, npix = (size_t)width * height;
        a = dmaps[(size_t)ch * npix + pix];
        b = dmaps[(size_t)(3 + ch) * npix + pix];
        e = dmaps[(size_t)(6 + ch) * npix + pix];
      }
      sm01[r][c] = make_float2(a, b);
      sm2[r][c] = e;
    }
    __syncthreads();
    // The blur of the three partial maps (loss.rs:124-127), blocked and streamed as in
    // ssim_fwd_kernel; zero-padded taps add +0.0 (the sums start at +0.0 and never become
    // -0.0).
    for (int item = tid; item < kLE * (kLT / kRB); item += kLossThreads) {
      const int r = item / (kLT / kRB), c0 = (item % (kLT / kRB)) * kRB;
      f2 a01[kRB];
      float a2[kRB];
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        a01[o] = f2_splat(0.0f);
        a2[o] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < kRB + 10; q++) {
        const float2 t = sm01[r][c0 + q];
        const f2 v = f2_make(t.x, t.y);
        const float e = sm2[r][c0 + q];
#pragma unroll
        for (int o = 0; o < kRB; o++) {
          const int k = q - o;
          if (k < 0 || k > 10) continue;
          a01[o] = f2_add(a01[o], f2_mul(wp[k], v));
          a2[o] += K.w[tap_weight(k)] * e;
        }
      }
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        float lo, hi;
        f2_split(a01[o], lo, hi);
        h01[r][c0 + o] = make_float2(lo, hi);
        h2[r][c0 + o] = a2[o];
      }
    }
    __syncthreads();
    for (int item = tid; item < kLT * (kLT / kRB); item += kLossThreads) {
      const int c = item % kLT, r0 = (item / kLT) * kRB;
      f2 b01[kRB];
      float b2[kRB];
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        b01[o] = f2_splat(0.0f);
        b2[o] = 0.0f;
      }
#pragma unroll
      for (int q = 0; q < kRB + 10; q++) {
        const float2 t = h01[r0 + q][c];
        const f2 v = f2_make(t.x, t.y);
        const float e = h2[r0 + q][c];
#pragma unroll
        for (int o = 0; o < kRB; o++) {
          const int k = q - o;
          if (k < 0 || k > 10) continue;
          b01[o] = f2_add(b01[o], f2_mul(wp[k], v));
          b2[o] += K.w[tap_weight(k)] * e;
        }
      }
#pragma unroll
      for (int o = 0; o < kRB; o++) {
        const int gy = oy0 + r0 + o, gx = ox0 + c;
        if (gx >= (int)width || gy >= (int)height) continue;
        float bmu, bexx;
        f2_split(b01[o], bmu, bexx);
        const float bexy = b2[o];
        const size_t idx = ((size_t)gy * width + gx) * 3 + ch;
        const float x = pred[idx];
        const float y = load_target(target, target_u8, idx);
        const float dssim = (bmu + 2.0f * x * bexx + y * bexy) * inv_n;
        const float d = x - y;
        const float sign = d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f);
        grad[idx] = (w1 * sign - lambda * dssim) * scale;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------------------
// Small views: a block takes one channel of a 32 x 16 tile, and each blur pass gives a thread
// kRun consecutive outputs of a row (then of a column) and streams their kRun + 10 inputs once.
// Such a view has too few 32 x 32 tiles of three channels for the SMs, so its time is one
// block's chain: 256x256 42 -> 18.5 us, 64x48 37 -> 12.6 us (runs of 8 outputs 22.6 and 18.5).
// ---------------------------------------------------------------------------------------
constexpr int kRun = 4;
constexpr int kTileW = kLossTile;
constexpr int kEdgeW = kTileW + 2 * kHalo;
constexpr int kTileH = 16, kEdgeH = kTileH + 2 * kHalo;
constexpr int kItemsH = kEdgeH * (kTileW / kRun), kItemsV = kTileW * (kTileH / kRun);
constexpr int kSmallThreads = (kItemsH + 31) / 32 * 32;
static_assert(kItemsV <= kSmallThreads, "a thread takes one run per pass");
// Row strides in shared memory: 8 rows of 16-byte accesses at one column hit distinct banks.
constexpr int kStride2 = 42, kStride1 = 44, kStrideH2 = 34, kStrideH1 = 36;
struct FwdTile {
  float2 xy[kEdgeH][kStride2];                            // (prediction, target)
  float2 h01[kEdgeH][kStrideH2], h23[kEdgeH][kStrideH2];  // horizontal blurs of (x, y), (x^2, y^2)
  float h4[kEdgeH][kStrideH1];                            // and of x y
  double red[3][kSmallThreads / 32];
};
struct BwdTile {
  float2 m01[kEdgeH][kStride2];  // partial maps w.r.t. mu_x and E[x^2]
  float m2[kEdgeH][kStride1];    // and w.r.t. E[xy]
  float2 h01[kEdgeH][kStrideH2];
  float h2[kEdgeH][kStrideH1];
  double red[3][kSmallThreads / 32];
};

// One tap of an output's running sums: acc[o] += w_k v for the outputs o that input q reaches.
// Both blur passes add their taps in window order (loss.rs:42-70) from +0.0; taps outside the
// image read the tile's zero padding and add +0.0, which leaves every sum as the reference's
// (it skips them).
__device__ __forceinline__ void tap2(f2 acc[kRun], const f2 w[6], int q, f2 v) {
#pragma unroll
  for (int o = 0; o < kRun; o++)
    if (q - o >= 0 && q - o <= 10) acc[o] = f2_add(acc[o], f2_mul(w[tap_weight(q - o)], v));
}
__device__ __forceinline__ void tap1(float acc[kRun], const LossKernel& K, int q, float v) {
#pragma unroll
  for (int o = 0; o < kRun; o++)
    if (q - o >= 0 && q - o <= 10) acc[o] += K.w[tap_weight(q - o)] * v;
}
__device__ __forceinline__ void store_run(float2* dst, const f2 a[kRun]) {
#pragma unroll
  for (int o = 0; o < kRun; o += 2) {
    float4 v;
    f2_split(a[o], v.x, v.y);
    f2_split(a[o + 1], v.z, v.w);
    *reinterpret_cast<float4*>(dst + o) = v;
  }
}
__device__ __forceinline__ void store_run(float* dst, const float a[kRun]) {
#pragma unroll
  for (int o = 0; o < kRun; o += 4) *reinterpret_cast<float4*>(dst + o) = make_float4(a[o], a[o + 1], a[o + 2], a[o + 3]);
}

// Per-pixel SSIM and its partial maps; the block's sums of SSIM, |x - y| and the squared
// clamped error (PSNR) go to partial[3 * block].
__global__ void __launch_bounds__(kSmallThreads) ssim_fwd_small_kernel(
    const float* __restrict__ pred, const void* __restrict__ target_arg, int target_u8, uint32_t width_arg,
    uint32_t height_arg, LossKernel K, float* __restrict__ dmaps, double* __restrict__ partial,
    const StepParams* __restrict__ sp) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char loss_smem[];
  FwdTile& t = *reinterpret_cast<FwdTile*>(loss_smem);
  const void* target = sp ? sp->target : target_arg;
  const int ox = blockIdx.x * kTileW, oy = blockIdx.y * kTileH;
  const int width = (int)width_arg, height = (int)height_arg, ch = blockIdx.z, tid = threadIdx.x;
  const float c1 = 0.01f * 0.01f, c2 = 0.03f * 0.03f;
  for (int i = tid; i < kEdgeH * kEdgeW; i += kSmallThreads) {
    const int r = i / kEdgeW, c = i % kEdgeW;
    const int gy = oy - kHalo + r, gx = ox - kHalo + c;
    float vx = 0.0f, vy = 0.0f;
    if (gx >= 0 && gx < width && gy >= 0 && gy < height) {
      const size_t idx = ((size_t)gy * width + gx) * 3 + ch;
      vx = pred[idx];
      vy = load_target(target, target_u8, idx);
    }
    t.xy[r][c] = make_float2(vx, vy);
  }
  f2 wp[6];
#pragma unroll
  for (int k = 0; k < 6; k++) wp[k] = f2_splat(K.w[k]);
  __syncthreads();
  // Horizontal pass (loss.rs:42-56) of every row with its halo.
  if (tid < kItemsH) {
    const int r = tid % kEdgeH, c0 = tid / kEdgeH * kRun;
    f2 a01[kRun], a23[kRun];
    float a4[kRun];
#pragma unroll
    for (int o = 0; o < kRun; o++) {
      a01[o] = a23[o] = f2_splat(0.0f);
      a4[o] = 0.0f;
    }
#pragma unroll
    for (int q = 0; q < kRun + 10; q += 2) {
      const float4 v = *reinterpret_cast<const float4*>(&t.xy[r][c0 + q]);
      const f2 va = f2_make(v.x, v.y), vb = f2_make(v.z, v.w);
      tap2(a01, wp, q, va);
      tap2(a23, wp, q, f2_mul(va, va));
      tap1(a4, K, q, v.x * v.y);
      tap2(a01, wp, q + 1, vb);
      tap2(a23, wp, q + 1, f2_mul(vb, vb));
      tap1(a4, K, q + 1, v.z * v.w);
    }
    store_run(&t.h01[r][c0], a01);
    store_run(&t.h23[r][c0], a23);
    store_run(&t.h4[r][c0], a4);
  }
  __syncthreads();
  // Vertical pass (loss.rs:58-70) and per-pixel SSIM (loss.rs:101-119).
  double s_ssim = 0.0, s_l1 = 0.0, s_se = 0.0;
  if (tid < kItemsV) {
    const int c = tid % kTileW, r0 = tid / kTileW * kRun;
    f2 m01[kRun], e23[kRun];
    float e4[kRun];
#pragma unroll
    for (int o = 0; o < kRun; o++) {
      m01[o] = e23[o] = f2_splat(0.0f);
      e4[o] = 0.0f;
    }
#pragma unroll
    for (int q = 0; q < kRun + 10; q++) {
      const float2 t01 = t.h01[r0 + q][c], t23 = t.h23[r0 + q][c];
      tap2(m01, wp, q, f2_make(t01.x, t01.y));
      tap2(e23, wp, q, f2_make(t23.x, t23.y));
      tap1(e4, K, q, t.h4[r0 + q][c]);
    }
    const int gx = ox + c;
    const size_t npix = (size_t)width * height;
#pragma unroll
    for (int o = 0; o < kRun; o++) {
      const int gy = oy + r0 + o;
      if (gx >= width || gy >= height) continue;
      float mx, my, exx, eyy;
      f2_split(m01[o], mx, my);
      f2_split(e23[o], exx, eyy);
      const float sx2 = exx - mx * mx;
      const float sy2 = eyy - my * my;
      const float sxy = e4[o] - mx * my;
      const float n1 = 2.0f * mx * my + c1;
      const float n2 = 2.0f * sxy + c2;
      const float d1 = mx * mx + my * my + c1;
      const float d2 = sx2 + sy2 + c2;
      const float num = n1 * n2;
      const float den = d1 * d2;
      const float sv = num / den;
      const float dn_dmx = 2.0f * my * n2 - 2.0f * my * n1;
      const float dd_dmx = 2.0f * mx * d2 - 2.0f * mx * d1;
      // The partial maps are planar (map, channel, pixel), so that the backward's tile loads are
      // contiguous.
      const size_t pix = (size_t)gy * width + gx;
      dmaps[(size_t)ch * npix + pix] = (dn_dmx * den - num * dd_dmx) / (den * den);
      dmaps[(size_t)(3 + ch) * npix + pix] = -num * d1 / (den * den);
      dmaps[(size_t)(6 + ch) * npix + pix] = 2.0f * n1 / den;
      const float2 xy = t.xy[r0 + o + kHalo][c + kHalo];
      s_ssim += (double)sv;
      s_l1 += (double)fabsf(xy.x - xy.y);
      const double e = (double)fminf(fmaxf(xy.x, 0.0f), 1.0f) - (double)fminf(fmaxf(xy.y, 0.0f), 1.0f);
      s_se += e * e;
    }
  }
  const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s_ssim += __shfl_xor_sync(0xffffffffu, s_ssim, o);
    s_l1 += __shfl_xor_sync(0xffffffffu, s_l1, o);
    s_se += __shfl_xor_sync(0xffffffffu, s_se, o);
  }
  if (lane == 0) {
    t.red[0][warp] = s_ssim;
    t.red[1][warp] = s_l1;
    t.red[2][warp] = s_se;
  }
  __syncthreads();
  if (tid < 3) {
    double v = 0.0;
    for (int w = 0; w < kSmallThreads / 32; w++) v += t.red[tid][w];
    const size_t block = ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * 3 + ch;
    partial[3 * block + tid] = v;
  }
}

// Gradient of the loss w.r.t. the prediction (loss.rs:124-133, :155-169); the first block also
// finishes the loss values.
__global__ void __launch_bounds__(kSmallThreads) ssim_bwd_small_kernel(
    const float* __restrict__ pred, const void* __restrict__ target_arg, int target_u8, uint32_t width_arg,
    uint32_t height_arg, LossKernel K, const float* __restrict__ dmaps, const double* __restrict__ partial,
    float lambda, float* __restrict__ grad, float* __restrict__ out3, const StepParams* __restrict__ sp) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char loss_smem[];
  BwdTile& t = *reinterpret_cast<BwdTile*>(loss_smem);
  if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    finalize_loss<kSmallThreads>(partial, 3 * gridDim.x * gridDim.y, 3 * (uint64_t)width_arg * height_arg, lambda,
                               t.red, out3);
  }
  const void* target = sp ? sp->target : target_arg;
  const int ox = blockIdx.x * kTileW, oy = blockIdx.y * kTileH;
  const int width = (int)width_arg, height = (int)height_arg, ch = blockIdx.z, tid = threadIdx.x;
  const size_t npix = (size_t)width * height;
  for (int i = tid; i < kEdgeH * kEdgeW; i += kSmallThreads) {
    const int r = i / kEdgeW, c = i % kEdgeW;
    const int gy = oy - kHalo + r, gx = ox - kHalo + c;
    float m0 = 0.0f, m1 = 0.0f, m2 = 0.0f;
    if (gx >= 0 && gx < width && gy >= 0 && gy < height) {
      const size_t pix = (size_t)gy * width + gx;
      m0 = dmaps[(size_t)ch * npix + pix];
      m1 = dmaps[(size_t)(3 + ch) * npix + pix];
      m2 = dmaps[(size_t)(6 + ch) * npix + pix];
    }
    t.m01[r][c] = make_float2(m0, m1);
    t.m2[r][c] = m2;
  }
  f2 wp[6];
#pragma unroll
  for (int k = 0; k < 6; k++) wp[k] = f2_splat(K.w[k]);
  __syncthreads();
  // The blur of the three partial maps (the blur is self-adjoint, loss.rs:124-127).
  if (tid < kItemsH) {
    const int r = tid % kEdgeH, c0 = tid / kEdgeH * kRun;
    f2 a01[kRun];
    float a2[kRun];
#pragma unroll
    for (int o = 0; o < kRun; o++) {
      a01[o] = f2_splat(0.0f);
      a2[o] = 0.0f;
    }
#pragma unroll
    for (int q = 0; q < kRun + 10; q += 2) {
      const float4 v = *reinterpret_cast<const float4*>(&t.m01[r][c0 + q]);
      const float2 e = *reinterpret_cast<const float2*>(&t.m2[r][c0 + q]);
      tap2(a01, wp, q, f2_make(v.x, v.y));
      tap1(a2, K, q, e.x);
      tap2(a01, wp, q + 1, f2_make(v.z, v.w));
      tap1(a2, K, q + 1, e.y);
    }
    store_run(&t.h01[r][c0], a01);
    store_run(&t.h2[r][c0], a2);
  }
  __syncthreads();
  if (tid < kItemsV) {
    const int c = tid % kTileW, r0 = tid / kTileW * kRun;
    f2 b01[kRun];
    float b2[kRun];
#pragma unroll
    for (int o = 0; o < kRun; o++) {
      b01[o] = f2_splat(0.0f);
      b2[o] = 0.0f;
    }
#pragma unroll
    for (int q = 0; q < kRun + 10; q++) {
      const float2 v = t.h01[r0 + q][c];
      tap2(b01, wp, q, f2_make(v.x, v.y));
      tap1(b2, K, q, t.h2[r0 + q][c]);
    }
    const float inv_n = 1.0f / (float)(npix * 3);
    const float w1 = (1.0f - lambda) * inv_n;
    const int gx = ox + c;
#pragma unroll
    for (int o = 0; o < kRun; o++) {
      const int gy = oy + r0 + o;
      if (gx >= width || gy >= height) continue;
      float bmu, bexx;
      f2_split(b01[o], bmu, bexx);
      const float bexy = b2[o];
      const size_t idx = ((size_t)gy * width + gx) * 3 + ch;
      const float x = pred[idx];
      const float y = load_target(target, target_u8, idx);
      const float dssim = (bmu + 2.0f * x * bexx + y * bexy) * inv_n;
      const float d = x - y;
      const float sign = d > 0.0f ? 1.0f : (d < 0.0f ? -1.0f : 0.0f);
      grad[idx] = w1 * sign - lambda * dssim;
    }
  }
}

LossKernel make_loss_kernel() {
  // gaussian_kernel (loss.rs:14-27), in f32 with the host libm, as the reference does.
  LossKernel k;
  const float sigma = 1.5f;
  float sum = 0.0f;
  float w[11];
  for (int i = 0; i < 11; i++) {
    const float x = (float)i - 5.0f;
    w[i] = expf(-(x * x) / (2.0f * sigma * sigma));
    sum += w[i];
  }
  for (int i = 0; i < 6; i++) k.w[i] = w[5 + i] / sum;
  return k;
}

Status launch_loss(Ctx* c, const float* pred, const void* target, int target_u8, uint32_t width, uint32_t height,
                   float lambda, float* grad, float* out3, const StepParams* sp, const BatchTable* bt,
                   uint32_t blocks_cap, uint64_t pix_cap) {
  // The line between the two: 32 x 32 tiles per SM. Below 4 the small kernels (640x480 39 us against
  // 58, 800x600 53 against 69); at 1297x840 (7.4) they are even (109 and 108 us) and at 1920x1080
  // (13.8) the large ones lead (192 against 211). A batch's table counts 32 x 32 tiles.
  const uint64_t tiles = (uint64_t)ceil_div(width, kLT) * ceil_div(height, kLT);
  const bool small = !bt && tiles < 4 * (uint64_t)c->sm_count;
  const dim3 grid = bt      ? dim3(blocks_cap)
                    : small ? dim3(ceil_div(width, kTileW), ceil_div(height, kTileH), 3)
                            : dim3(ceil_div(width, kLT), ceil_div(height, kLT));
  float* dmaps = nullptr;
  double* sums = nullptr;
  SPLAT_TRY(arena_reserve(c, (bt ? (size_t)pix_cap : (size_t)width * height) * 36, (void**)&dmaps));
  SPLAT_TRY(arena_reserve(c, (size_t)grid.x * grid.y * grid.z * 3 * 8, (void**)&sums));
  const LossKernel K = make_loss_kernel();
  if (small) {
    static_assert(sizeof(FwdTile) <= 48 * 1024 && sizeof(BwdTile) <= 48 * 1024, "");
    SPLAT_TRY(launch_chained(c, "ssim_fwd_small_kernel", ssim_fwd_small_kernel, grid, kSmallThreads, sizeof(FwdTile),
                             pred, target, target_u8, width, height, K, dmaps, sums, sp));
    SPLAT_TRY(launch_chained(c, "ssim_bwd_small_kernel", ssim_bwd_small_kernel, grid, kSmallThreads, sizeof(BwdTile),
                             pred, target, target_u8, width, height, K, dmaps, sums, lambda, grad, out3, sp));
  } else {
    SPLAT_TRY(launch_chained(c, "ssim_fwd_kernel", ssim_fwd_kernel, grid, kLossThreads, 0, pred, target, target_u8,
                             width, height, K, dmaps, sums, sp, bt));
    SPLAT_TRY(launch_chained(c, "ssim_bwd_kernel", ssim_bwd_kernel, grid, kLossThreads, 0, pred, target, target_u8,
                             width, height, K, dmaps, sums, lambda, grad, out3, sp, bt));
  }
  return Status::ok();
}

}  // namespace splat
