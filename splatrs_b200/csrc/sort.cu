// Binning (reference src/rasterize.rs:60-128) on the device:
//   scan of per-Gaussian tile counts -> entry offsets (Binning::entry_offset),
//   warp-cooperative emission of one (tile | depth) key per entry in Gaussian order,
//   stable LSD radix sort of the keys carrying the Gaussian index,
//   per-tile [start, end) ranges.
//
// Keys are compacted before sorting: the reference key is (tile << 32) | depth_bits with
// depth_bits the f32 bits of a positive depth. Subtracting the smallest visible depth bits
// and packing the tile above the remaining significant bits keeps the order of every pair
// of keys, so the sort runs over ceil((tile bits + depth bits) / 8) passes instead of 8.
// The sort is stable, and entries enter it in entry order, which reproduces the
// reference's tie-break on the entry index.
#include <mutex>
#include <set>
#include <utility>

#include "common.cuh"
#include "kernels.cuh"

namespace splat {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096 values per block

// ---------------------------------------------------------------------------------------
// Exclusive scan of uint32 counts into uint32 offsets (with the total written at [n]): sums of
// blocks of 4,096 values, then every block adds up the sums before it and scans its own. Up to
// kScanDirect blocks that costs a block at most kScanDirect reads of L2 and saves a launch (n =
// 1M: 9.4 us for two kernels against 14.7 for three with 4-byte loads; 10,000: 6.1 against 9.3);
// longer inputs scan the sums in between.
// Totals are carried in 64 bits.
// ---------------------------------------------------------------------------------------
constexpr uint32_t kScanDirect = 1024;
__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v, uint64_t* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  uint64_t t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  return t;  // valid in thread 0
}

// Block-wide exclusive scan of one uint64 per thread; returns the exclusive prefix, and
// the block total through *total.
__device__ __forceinline__ uint64_t block_exclusive_u64(uint64_t v, uint64_t* sh, uint64_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  uint64_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint64_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sh[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint64_t w = lane < nw ? sh[lane] : 0;
    uint64_t wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint64_t y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < nw) sh[lane] = wi - w;
    if (lane == nw - 1) sh[32] = wi;
  }
  __syncthreads();
  uint64_t r = sh[warp] + incl - v;
  *total = sh[32];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t* __restrict__ in, int64_t n,
                                                                   uint64_t* __restrict__ partial) {
  chain_begin();
  __shared__ uint64_t sh[33];
  const int64_t base = (int64_t)blockIdx.x * kScanTile;
  uint64_t s = 0;
#pragma unroll
  for (int j = 0; j < kScanItems; j++) {
    const int64_t idx = base + (int64_t)j * kScanThreads + threadIdx.x;
    if (idx < n) s += in[idx];
  }
  s = block_sum_u64(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// Single block: exclusive scan of `m` partials in place; total to *total.
__global__ void __launch_bounds__(1024) scan_partials_kernel(uint64_t* __restrict__ partial, int64_t m,
                                                             uint64_t* __restrict__ total) {
  chain_begin();
  __shared__ uint64_t sh[33];
  uint64_t carry = 0;
  for (int64_t base = 0; base < m; base += blockDim.x) {
    const int64_t idx = base + threadIdx.x;
    const uint64_t v = idx < m ? partial[idx] : 0;
    uint64_t tot;
    const uint64_t ex = block_exclusive_u64(v, sh, &tot);
    if (idx < m) partial[idx] = carry + ex;
    carry += tot;
  }
  if (threadIdx.x == 0) *total = carry;
}

// Writes out[i] = exclusive prefix (uint32) for i < n, and, from the last block, the total to
// *total, out[n] (with write_total) and *host_total (mapped host memory, may be NULL). `scanned`:
// partial holds prefixes, else the blocks' sums. A thread takes 16 consecutive values, as four
// 16-byte loads and stores where the pointers allow.
__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const uint32_t* __restrict__ in, int64_t n,
                                                                  const uint64_t* __restrict__ partial, int scanned,
                                                                  uint64_t* __restrict__ total,
                                                                  uint32_t* __restrict__ out, int write_total,
                                                                  volatile uint64_t* host_total) {
  chain_begin();
  __shared__ uint64_t sh[33];
  __shared__ uint64_t before;
  uint64_t first = 0;
  if (scanned) {
    first = partial[blockIdx.x];
  } else {
    for (uint32_t k = threadIdx.x; k < blockIdx.x; k += kScanThreads) first += partial[k];
    first = block_sum_u64(first, sh);
    if (threadIdx.x == 0) before = first;
    __syncthreads();
    first = before;
  }
  const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kScanItems;
  uint32_t v[kScanItems];
  uint64_t s = 0;
  const bool whole = base + kScanItems <= n;
  if (whole && (reinterpret_cast<uintptr_t>(in) & 15u) == 0) {
    const uint4* in4 = reinterpret_cast<const uint4*>(in + base);
#pragma unroll
    for (int j = 0; j < kScanItems / 4; j++) {
      const uint4 q = in4[j];
      v[4 * j] = q.x;
      v[4 * j + 1] = q.y;
      v[4 * j + 2] = q.z;
      v[4 * j + 3] = q.w;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kScanItems; j++) v[j] = base + j < n ? in[base + j] : 0u;
  }
#pragma unroll
  for (int j = 0; j < kScanItems; j++) s += v[j];
  uint64_t tot;
  uint64_t run = first + block_exclusive_u64(s, sh, &tot);
#pragma unroll
  for (int j = 0; j < kScanItems; j++) {
    const uint32_t c = v[j];
    v[j] = (uint32_t)run;
    run += c;
  }
  if (whole && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
    uint4* out4 = reinterpret_cast<uint4*>(out + base);
#pragma unroll
    for (int j = 0; j < kScanItems / 4; j++) out4[j] = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  } else {
#pragma unroll
    for (int j = 0; j < kScanItems; j++)
      if (base + j < n) out[base + j] = v[j];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    const uint64_t all = first + tot;
    *total = all;
    if (write_total) out[n] = (uint32_t)all;
    if (host_total) {
      *host_total = all;
      __threadfence_system();
    }
  }
}

// The visible depths' range before a projection: (smallest, largest) = (0xffffffff, 0).
__global__ void reset_range_kernel(uint32_t* __restrict__ range) {
  chain_begin(); range[threadIdx.x] = threadIdx.x ? 0u : 0xffffffffu; }

Status launch_reset_range(Ctx* c, uint32_t* range) {
  SPLAT_TRY(launch_chained(c, "reset_range_kernel", reset_range_kernel, 1, 2, 0, range));
  return Status::ok();
}

__global__ void fill_u32_kernel(uint32_t* __restrict__ dst, size_t words, uint32_t value, int vector) {
  chain_begin();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t quads = vector ? words / 4 : 0;
  uint4* d4 = reinterpret_cast<uint4*>(dst);
  const uint4 v4 = make_uint4(value, value, value, value);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += stride) d4[i] = v4;
  for (size_t i = quads * 4 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) dst[i] = value;
}

// Zeroes up to three regions of 32-bit words in one launch, and stores two words of `show` (may
// be NULL) into mapped host memory on the way.
__global__ void zero3_u32_kernel(uint32_t* __restrict__ a, size_t na, uint32_t* __restrict__ b, size_t nb,
                                 uint32_t* __restrict__ c3, size_t nc, const uint32_t* __restrict__ show,
                                 volatile uint32_t* host) {
  chain_begin();
  if (show && blockIdx.x == 0 && threadIdx.x < 2) {
    host[threadIdx.x] = show[threadIdx.x];
    __threadfence_system();
  }
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < na + nb + nc; i += stride) {
    if (i < na)
      a[i] = 0u;
    else if (i < na + nb)
      b[i - na] = 0u;
    else
      c3[i - na - nb] = 0u;
  }
}

static Status launch_zero3_u32(Ctx* c, void* a, size_t na, void* b, size_t nb, void* c3, size_t nc,
                               const uint32_t* show = nullptr) {
  const size_t words = na + nb + nc;
  if (words == 0) return Status::ok();
  const uint32_t grid = (uint32_t)std::min<size_t>((words + 255) / 256, (size_t)c->sm_count * 8);
  SPLAT_TRY(launch_chained(c, "zero3_u32_kernel", zero3_u32_kernel, grid, 256, 0, static_cast<uint32_t*>(a), na,
                           static_cast<uint32_t*>(b), nb, static_cast<uint32_t*>(c3), nc, show,
                           static_cast<volatile uint32_t*>(c->host_small_dev)));
  return Status::ok();
}

Status launch_fill_u32(Ctx* c, void* dst, size_t words, uint32_t value) {
  if (words == 0) return Status::ok();
  const int vector = (reinterpret_cast<uintptr_t>(dst) & 15u) == 0;
  const size_t items = vector ? (words + 3) / 4 : words;
  const uint32_t grid = (uint32_t)std::min<size_t>((items + 255) / 256, (size_t)c->sm_count * 8);
  SPLAT_TRY(launch_chained(c, "fill_u32_kernel", fill_u32_kernel, grid, 256, 0, reinterpret_cast<uint32_t*>(dst),
                           words, value, vector));
  return Status::ok();
}

__global__ void publish_u32_kernel(const uint32_t* __restrict__ a, int na, const uint32_t* __restrict__ b, int nb,
                                   volatile uint32_t* out) {
  chain_begin();
  const int lane = threadIdx.x;
  if (lane < na) out[lane] = a[lane];
  if (lane < nb) out[na + lane] = b[lane];
  __threadfence_system();
}

__global__ void load_words_kernel(const volatile uint32_t* src, uint32_t* __restrict__ dst, int words) {
  chain_begin();
  for (int i = threadIdx.x; i < words; i += 32) dst[i] = src[i];
}

Status launch_load_words(Ctx* c, const void* src_mapped_dev, void* dst, int words) {
  SPLAT_TRY(launch_chained(c, "load_words_kernel", load_words_kernel, 1, 32, 0,
                           static_cast<const volatile uint32_t*>(src_mapped_dev), static_cast<uint32_t*>(dst),
                           words));
  return Status::ok();
}

Status launch_publish_u32(Ctx* c, const uint32_t* a, int na, const uint32_t* b, int nb) {
  return launch_publish_u32_to(c, a, na, b, nb, c->host_small_dev);
}

Status launch_publish_u32_to(Ctx* c, const uint32_t* a, int na, const uint32_t* b, int nb, void* out_dev) {
  if (na < 0 || nb < 0 || na + nb > 32) return Status::make(SPLAT_ERR_INVALID, "publish: at most 32 words");
  SPLAT_TRY(launch_chained(c, "publish_u32_kernel", publish_u32_kernel, 1, 32, 0, a, na, b, nb,
                           reinterpret_cast<volatile uint32_t*>(out_dev)));
  return Status::ok();
}

Status take_sort_error(Ctx* c) {
  volatile uint32_t* w = reinterpret_cast<volatile uint32_t*>(c->host_small) + kSortErrWord;
  if (*w == 0) return Status::ok();
  *w = 0;
  return Status::make(SPLAT_ERR_TIMEOUT, "radix sort: a tile's look-back wait ran out; that sort's output is invalid");
}

Status launch_scan_u32_into(Ctx* c, const uint32_t* in, int64_t n, uint32_t* out, int write_total, uint64_t* partial,
                            uint64_t* total, uint64_t* host_total) {
  const uint32_t blocks = ceil_div((uint64_t)std::max<int64_t>(n, 1), kScanTile);
  const int scanned = blocks > kScanDirect;
  if (blocks > 1) {
    SPLAT_TRY(launch_chained(c, "scan_reduce_kernel", scan_reduce_kernel, blocks, kScanThreads, 0, in, n, partial));
  }
  if (scanned) {
    SPLAT_TRY(launch_chained(c, "scan_partials_kernel", scan_partials_kernel, 1, 1024, 0, partial, blocks, total));
  }
  SPLAT_TRY(launch_chained(c, "scan_apply_kernel", scan_apply_kernel, blocks, kScanThreads, 0, in, n, partial,
                           scanned, total, out, write_total, host_total));
  return Status::ok();
}

Status launch_scan_u32(Ctx* c, const uint32_t* in, int64_t n, uint32_t* out, int write_total, uint64_t* total_dev,
                       uint64_t* host_total) {
  uint64_t* partial = nullptr;
  SPLAT_TRY(arena_reserve(c, (size_t)ceil_div((uint64_t)std::max<int64_t>(n, 1), kScanTile) * 8, (void**)&partial));
  return launch_scan_u32_into(c, in, n, out, write_total, partial, total_dev, host_total);
}

// ---------------------------------------------------------------------------------------
// Sort keys. A key holds, from the top: the tile, the depth bits above the smallest visible
// ones (dbits of them) and, when all three fit in 64 bits ("packed"), the entry's Gaussian in
// vbits low bits, which the sort does not look at. Otherwise the Gaussian travels beside the
// key. Packed keys take 16 bytes of traffic per entry and pass instead of 24 and half the
// registers.
// ---------------------------------------------------------------------------------------
constexpr int kMaxPasses = 8;
struct KeyLayout {
  int64_t E;  // entries to sort
  int dbits, vbits, passes;
};

inline int bits_for(uint64_t values) {  // bits that tell `values` values apart
  return values <= 1 ? 0 : 64 - __builtin_clzll(values - 1);
}

// ---------------------------------------------------------------------------------------
// Key emission (rasterize.rs:76-104): the entries of Gaussian g occupy
// [entry_offset[g], entry_offset[g+1]) and enumerate its tile rectangle row by row. A warp takes
// 32 consecutive Gaussians at a time and writes their entries contiguously; the digits of all
// passes are counted on the way (per-block counters in shared memory, native integer atomics,
// added to the global ones once per block; the grid is a few blocks per SM so that this stays
// small). 3.08M entries: 27 us against 17 and 15 for emission and a counting kernel, and one launch
// less.
// ---------------------------------------------------------------------------------------
template <bool kPacked>
__device__ __forceinline__ void emit_keys_body(const float4* __restrict__ rec, const uint32_t* __restrict__ entry_offset,
                                               int64_t n, uint32_t tiles_x, const uint32_t* __restrict__ depth_range,
                                               const KeyLayout lay, int64_t limit, uint64_t* __restrict__ keys,
                                               uint32_t* __restrict__ vals, uint32_t* __restrict__ hist,
                                               const BatchTable* bt, int64_t n_view) {
  __shared__ uint32_t cnt_sh[kMaxPasses][256];
  for (int i = threadIdx.x; i < lay.passes * 256; i += blockDim.x) cnt_sh[i >> 8][i & 255] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t first = ((((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5)) * 32; first < n; first += warps * 32) {
    const int64_t g = first + lane;
    uint32_t cnt = 0, tx0 = 0, ty0 = 0, w = 1, dkey = 0, toff = 0, txs = tiles_x, o0 = 0;
    if (g < n) {
      if (bt) {  // batch: the record's view sets its tile grid and first global tile
        const int v = (int)(g / n_view);
        toff = bt->tile_start[v];
        txs = bt->tiles_x[v];
      }
      o0 = entry_offset[g];
      cnt = entry_offset[g + 1] - o0;
      if (cnt) {
        const float4 r3 = rec[4 * g + 3];
        const uint32_t tmin = fbits(r3.z), tmax = fbits(r3.w);
        tx0 = tmin & 0xffffu;
        ty0 = tmin >> 16;
        w = (tmax & 0xffffu) - tx0;
        dkey = fbits(r3.x) - depth_range[0];
      }
    }
    const uint32_t start = __shfl_sync(0xffffffffu, o0, 0);
    // Inclusive warp scan of the counts.
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
    for (uint32_t j0 = 0; j0 < total; j0 += 32) {
      const uint32_t j = j0 + lane;
      // Owner lane: first lane whose inclusive count exceeds j (binary search over lanes).
      int lo = 0;
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const uint32_t v = __shfl_sync(0xffffffffu, incl, lo + step - 1);
        if (v <= j) lo += step;
      }
      const uint32_t o_incl = __shfl_sync(0xffffffffu, incl, lo);
      const uint32_t o_cnt = __shfl_sync(0xffffffffu, cnt, lo);
      const uint32_t o_tx0 = __shfl_sync(0xffffffffu, tx0, lo);
      const uint32_t o_ty0 = __shfl_sync(0xffffffffu, ty0, lo);
      const uint32_t o_w = __shfl_sync(0xffffffffu, w, lo);
      const uint32_t o_dkey = __shfl_sync(0xffffffffu, dkey, lo);
      uint32_t o_toff = 0, o_txs = tiles_x;
      if (bt) {
        o_toff = __shfl_sync(0xffffffffu, toff, lo);
        o_txs = __shfl_sync(0xffffffffu, txs, lo);
      }
      if (j < total && (int64_t)start + j < limit) {
        const uint32_t local = j - (o_incl - o_cnt);
        const uint32_t row = local / o_w;
        const uint32_t ty = o_ty0 + row, tx = o_tx0 + (local - row * o_w);
        const uint64_t tile = (uint64_t)o_toff + (uint64_t)ty * o_txs + tx;
        uint64_t key = (tile << lay.dbits) | (uint64_t)o_dkey;
        for (int p = 0; p < lay.passes; p++) atomicAdd(&cnt_sh[p][(uint32_t)(key >> (8 * p)) & 0xffu], 1u);
        const uint32_t gauss = (uint32_t)(first + lo);
        if (kPacked) {
          keys[start + j] = (key << lay.vbits) | gauss;
        } else {
          keys[start + j] = key;
          vals[start + j] = gauss;
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < lay.passes * 256; i += blockDim.x) {
    const uint32_t v = cnt_sh[i >> 8][i & 255];
    if (v) atomicAdd(&hist[i], v);
  }
}

template <bool kPacked>
__global__ void __launch_bounds__(256) emit_keys_kernel(const float4* __restrict__ rec,
                                                        const uint32_t* __restrict__ entry_offset, int64_t n,
                                                        uint32_t tiles_x, const uint32_t* __restrict__ depth_range,
                                                        KeyLayout lay, uint64_t* __restrict__ keys,
                                                        uint32_t* __restrict__ vals, uint32_t* __restrict__ hist) {
  chain_begin();
  emit_keys_body<kPacked>(rec, entry_offset, n, tiles_x, depth_range, lay, lay.E, keys, vals, hist, nullptr, 1);
}

// Passes that keys can need: depth bits span 32 bits at most (31 while depths are positive).
static int max_passes(int tbits) { return (tbits + 32 + 7) / 8; }

// Blocks of an emission over n records.
static uint32_t emit_blocks(const Ctx* c, int64_t n) {
  return (uint32_t)std::min<uint64_t>(ceil_div((uint64_t)n, 256), (uint64_t)c->sm_count * 6);
}

// ---------------------------------------------------------------------------------------
// Stable LSD radix sort, 8-bit digits, one kernel per pass (onesweep).
// The emission has counted every pass's digits. Each pass kernel takes tiles of keys in ticket
// order (an atomic counter, so a tile only ever waits for tiles whose blocks already run): each
// warp ranks 32 ROUNDS consecutive keys in rounds of 32 (position order) with match-any peer
// groups and per-warp digit counters; a per-digit prefix over the warps gives block-local stable
// ranks. The tile's global offset per digit is the digit's start (a prefix over the pass's
// histogram) plus the counts of that digit in all earlier tiles, found by decoupled look-back:
// every tile publishes its count per digit as soon as it has it (AGGREGATE), then its inclusive
// prefix (PREFIX); a tile walks back over its predecessors' words, adding aggregates until it
// meets a prefix. Every wait on a predecessor is bounded: past kLookbackSpins polls the tile sets
// the error bit 2 in *err, sets the abort word so no other tile waits any longer, and writes
// nothing (callers treat the sort as failed).
// ---------------------------------------------------------------------------------------
// Tile shapes by the number of keys. A pass is a chain (load, rounds, look-back, reorder, write)
// per block with a quarter to a half of the issue slots used and L2 at 10%, so small sorts take
// small tiles that spread over the SMs and large ones blocks with more warps. Per pass: 30k keys
// 5.6 us with 1,024-key tiles, 6.0 with 2,048, 7.6 with 4,096; 105k keys 6.9, 6.1, 7.1; 228k keys
// 9.4, 8.1, 9.5; 1.01M keys 21.5, 16.6, 15.0; 3.08M keys 36.8 with 2,048 and 36.2 with 4,096 (41.4
// before: 256 x 16 with the Gaussian beside the key and 128 registers; 512 x 16 35.3, 1,024 x 4
// 40.7). A look-back window of 32 words instead of 16 made the large pass 45.9 us.
template <int THREADS, int ROUNDS>
struct SortShape {
  static constexpr int kThreads = THREADS, kRounds = ROUNDS, kTile = THREADS * ROUNDS;
};
typedef SortShape<256, 4> SortSmall;
typedef SortShape<256, 8> SortMid;
typedef SortShape<512, 8> SortLarge;
constexpr int64_t kSmallSortKeys = 1 << 16, kMidSortKeys = 3 << 18;
inline uint64_t sort_tiles(int64_t keys) {
  return ceil_div((uint64_t)keys, keys <= kSmallSortKeys ? SortSmall::kTile
                                  : keys <= kMidSortKeys ? SortMid::kTile
                                                         : SortLarge::kTile);
}
constexpr uint32_t kLookbackSpins = 1u << 22;
constexpr int kLbWindow = 16;

// A look-back word: two flag bits (1 aggregate, 2 prefix) above the count. 32-bit words while
// every count fits in 30 bits, else 64-bit ones.
template <typename W>
struct LookbackWord {
  static constexpr int kShift = 8 * sizeof(W) - 2;
  static constexpr W kAggregate = (W)1 << kShift, kPrefix = (W)2 << kShift, kCount = ((W)1 << kShift) - 1;
};
inline bool wide_words(int64_t keys) { return keys >= (1ll << 30); }

// Control words of one sort (zeroed before it): the digit histogram of every pass, one
// ticket counter per pass, the abort word, and per pass one look-back word per tile and digit.
struct SortCtl {
  uint32_t* hist;    // [kMaxPasses][256]
  uint32_t* ticket;  // [kMaxPasses]
  uint32_t* abort;   // [1]
  void* status;      // [kMaxPasses][tiles][256] words
};
inline size_t status_bytes(int64_t keys, int passes) {
  return (size_t)passes * sort_tiles(keys) * 256 * (wide_words(keys) ? 8 : 4);
}
constexpr size_t kSortCounterWords = (size_t)kMaxPasses * 256 + kMaxPasses + 2;
inline size_t sort_ctl_bytes(int64_t keys) { return status_bytes(keys, kMaxPasses) + kSortCounterWords * 4 + 64; }
inline SortCtl carve_sort_ctl(void* base, int64_t keys) {
  SortCtl ctl;
  char* b = static_cast<char*>(base);
  ctl.status = b;
  b += status_bytes(keys, kMaxPasses);
  ctl.hist = reinterpret_cast<uint32_t*>(b);
  ctl.ticket = ctl.hist + (size_t)kMaxPasses * 256;
  ctl.abort = ctl.ticket + kMaxPasses;
  return ctl;
}

// What a pass writes: keys (and, unpacked, the Gaussians) for the next pass, or, from the last
// one, the sorted Gaussians, their tiles and (optional) the reference's 64-bit keys.
struct PassOut {
  uint64_t* keys;
  uint32_t* vals;
  uint32_t* tiles;
  uint64_t* ref_keys;
  uint32_t depth_min;
  int vbits, dbits;
  bool last;
};

// Dynamic shared memory of a pass: the tile's keys (and Gaussians) reordered by digit, the
// per-warp digit counters, the digits' block starts and output offsets, scan scratch.
template <typename S, bool kPacked>
constexpr size_t onesweep_smem() {
  return (size_t)S::kTile * (kPacked ? 8 : 12) + (size_t)(S::kThreads / 32) * 256 * 4 + 2 * 256 * 4 + 64;
}

// Exclusive prefix over the 256 digits of v (thread d < 256 holds digit d's value); `wsum` holds
// 8 words. Returns thread d's prefix.
__device__ __forceinline__ uint32_t digit_exclusive(uint32_t v, uint32_t* wsum) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();
  if (lane == 31 && warp < 8) wsum[warp] = incl;
  __syncthreads();
  uint32_t wprefix = 0;
#pragma unroll
  for (int w = 0; w < 7; w++)
    if (w < warp) wprefix += wsum[w];
  return wprefix + incl - v;
}

// One pass over keys_in[0, n) (digit at `shift`): `hist` is this pass's 256 global counts,
// `status` its look-back words, `ticket` its tile counter.
template <typename S, bool kPacked, typename W>
__device__ __forceinline__ void onesweep_body(const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in,
                                              int64_t n, int shift, const uint32_t* __restrict__ hist,
                                              W* __restrict__ status, uint32_t* __restrict__ ticket,
                                              uint32_t* __restrict__ abort_word, uint32_t* __restrict__ err,
                                              const PassOut& out, unsigned char* dsm) {
  typedef LookbackWord<W> LB;
  constexpr int TILE = S::kTile, ROUNDS = S::kRounds, WARPS = S::kThreads / 32;
  uint64_t* sk = reinterpret_cast<uint64_t*>(dsm);
  uint32_t* sv = reinterpret_cast<uint32_t*>(sk + TILE);
  uint32_t(*wcnt)[256] = reinterpret_cast<uint32_t(*)[256]>(sv + (kPacked ? 0 : TILE));
  uint32_t* dstart = reinterpret_cast<uint32_t*>(wcnt) + WARPS * 256;
  uint32_t* doff = dstart + 256;
  uint32_t* wsum = doff + 256;  // 8 words, then the tile number and the failure word
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tiles = (n + TILE - 1) / TILE;
  if (threadIdx.x == 0) {
    wsum[8] = atomicAdd(ticket, 1u);
    wsum[9] = 0;
  }
  for (int d = lane; d < 256; d += 32) wcnt[warp][d] = 0;
  __syncthreads();
  const uint32_t tile = wsum[8];
  if ((int64_t)tile >= tiles) return;
  const int64_t bbase = (int64_t)tile * TILE;
  const int64_t wbase = bbase + (int64_t)warp * (32 * ROUNDS);
  uint64_t k[ROUNDS];
  uint32_t v[kPacked ? 1 : ROUNDS];
  uint32_t rank[ROUNDS];
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const int64_t idx = wbase + r * 32 + lane;
    k[r] = idx < n ? keys_in[idx] : 0;
    if (!kPacked) v[kPacked ? 0 : r] = idx < n ? vals_in[idx] : 0u;
  }
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const bool valid = wbase + r * 32 + lane < n;
    const uint32_t d = valid ? ((uint32_t)(k[r] >> shift) & 0xffu) : 256u;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const uint32_t before = valid ? wcnt[warp][d] : 0u;
    rank[r] = before + __popc(peers & lt);
    __syncwarp();
    if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = before + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // Per digit (thread d): exclusive prefix over the warps and the tile's count.
  const int d = threadIdx.x;
  uint32_t total = 0, ghist = 0;
  W excl = 0;
  if (d < 256) {
    ghist = hist[d];
#pragma unroll
    for (int w = 0; w < WARPS; w++) {
      const uint32_t c = wcnt[w][d];
      wcnt[w][d] = total;
      total += c;
    }
    // Publish the tile's count of digit d at once; tile 0's is already its prefix.
    volatile W* my_word = status + (size_t)tile * 256 + d;
    *my_word = (tile == 0 ? LB::kPrefix : LB::kAggregate) | (W)total;
    // Look back over the earlier tiles, kLbWindow words at a time (independent loads), nearest
    // first: add aggregates until a prefix; a word not yet published is polled alone (bounded).
    bool failed = false;
    int64_t t = (int64_t)tile - 1;
    while (t >= 0) {
      W w[kLbWindow];
#pragma unroll
      for (int i = 0; i < kLbWindow; i++)
        w[i] = t - i >= 0 ? *(const volatile W*)(status + (size_t)(t - i) * 256 + d) : LB::kPrefix;
      int i = 0;
      bool done = false;
#pragma unroll
      for (int q = 0; q < kLbWindow; q++) {
        if (done || i < q) continue;  // stopped at a prefix or an unpublished word before q
        const W sq = w[q];
        if ((sq >> LB::kShift) == 0) continue;
        excl += sq & LB::kCount;
        i = q + 1;
        if ((sq >> LB::kShift) == 2) done = true;
      }
      if (done) break;
      t -= i;
      if (i == kLbWindow) continue;
      // Word t is not published yet: wait for it.
      const volatile W* wp = status + (size_t)t * 256 + d;
      uint32_t spins = 0;
      while ((*wp >> LB::kShift) == 0) {
        if (++spins >= kLookbackSpins || *(volatile uint32_t*)abort_word) {
          failed = true;
          break;
        }
        __nanosleep(32);
      }
      if (failed) break;
    }
    if (failed) {
      atomicOr(abort_word, 1u);
      // A plain store: err may be mapped host memory. Racing writers all set the same bit.
      volatile uint32_t* e = err;
      *e = *e | 2u;
      wsum[9] = 1;
    } else if (tile > 0) {
      *my_word = LB::kPrefix | (excl + (W)total);
    }
  }
  // Block starts of the digits and the pass's global digit starts.
  const uint32_t start = digit_exclusive(total, wsum);
  const uint32_t gstart = digit_exclusive(ghist, wsum);
  if (d < 256) {
    dstart[d] = start;
    doff[d] = gstart + (uint32_t)excl - start;  // output index = doff[digit] + block-sorted index
  }
  __syncthreads();
  if (wsum[9]) return;
  // Reorder the tile's keys by digit in shared memory (stable).
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    if (wbase + r * 32 + lane < n) {
      const uint32_t dg = (uint32_t)(k[r] >> shift) & 0xffu;
      const uint32_t pos = dstart[dg] + wcnt[warp][dg] + rank[r];
      sk[pos] = k[r];
      if (!kPacked) sv[pos] = v[kPacked ? 0 : r];
    }
  }
  __syncthreads();
  // Write out runs of equal digits contiguously.
  const int nb = (int)(n - bbase < TILE ? n - bbase : TILE);
  for (int i = threadIdx.x; i < nb; i += S::kThreads) {
    const uint64_t key = sk[i];
    const uint32_t pos = doff[(uint32_t)(key >> shift) & 0xffu] + (uint32_t)i;
    if (pos >= (uint64_t)n) continue;
    if (!out.last) {
      out.keys[pos] = key;
      if (!kPacked) out.vals[pos] = sv[i];
    } else {
      const uint64_t td = kPacked ? key >> out.vbits : key;  // tile | depth
      out.vals[pos] = kPacked ? (uint32_t)(key & ((1ull << out.vbits) - 1ull)) : sv[i];
      const uint32_t tl = (uint32_t)(td >> out.dbits);
      out.tiles[pos] = tl;
      if (out.ref_keys)
        out.ref_keys[pos] = ((uint64_t)tl << 32) | ((uint32_t)(td & ((1ull << out.dbits) - 1ull)) + out.depth_min);
    }
  }
}

template <typename S, bool kPacked, typename W>
__global__ void __launch_bounds__(S::kThreads) radix_onesweep_kernel(const uint64_t* __restrict__ keys_in,
                                                                     const uint32_t* __restrict__ vals_in, int64_t n,
                                                                     int pass, SortCtl ctl, uint32_t* __restrict__ err,
                                                                     PassOut out) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char dsm[];
  const uint64_t tiles = (uint64_t)((n + S::kTile - 1) / S::kTile);
  onesweep_body<S, kPacked, W>(keys_in, vals_in, n, 8 * pass + out.vbits, ctl.hist + 256 * pass,
                               static_cast<W*>(ctl.status) + (size_t)pass * tiles * 256, ctl.ticket + pass, ctl.abort,
                               err, out, dsm);
}

// Tile ranges (rasterize.rs:108-119) from the sorted entries' tiles (16-byte aligned): a thread
// takes four entries with one load and sees its neighbours' through the warp (3.08M entries: 11.5 ->
// 4.6 us).
constexpr int kRangeThreads = 256;
__device__ __forceinline__ void tile_ranges_body(const uint32_t* __restrict__ tiles, int64_t n,
                                                 uint32_t* __restrict__ ranges) {
  const int64_t i0 = 4 * ((int64_t)blockIdx.x * kRangeThreads + threadIdx.x);
  if ((i0 & ~(int64_t)127) >= n) return;  // the warp is past the end
  const uint32_t lane = threadIdx.x & 31;
  uint32_t t[4];
  if (i0 + 4 <= n) {
    const uint4 q = *reinterpret_cast<const uint4*>(tiles + i0);
    t[0] = q.x;
    t[1] = q.y;
    t[2] = q.z;
    t[3] = q.w;
  } else {
#pragma unroll
    for (int j = 0; j < 4; j++) t[j] = i0 + j < n ? tiles[i0 + j] : 0xffffffffu;  // no tile has this number
  }
  uint32_t prev = __shfl_up_sync(0xffffffffu, t[3], 1);
  if (lane == 0) prev = i0 > 0 ? tiles[i0 - 1] : 0xffffffffu;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const int64_t i = i0 + j;
    if (i <= n && t[j] != prev) {  // entry i starts its tile and ends the one before
      if (i < n) ranges[2 * (size_t)t[j]] = (uint32_t)i;
      if (i > 0 && prev != 0xffffffffu) ranges[2 * (size_t)prev + 1] = (uint32_t)i;
    }
    prev = t[j];
  }
  if (i0 + 4 == n) ranges[2 * (size_t)t[3] + 1] = (uint32_t)n;
}
__global__ void __launch_bounds__(kRangeThreads) tile_ranges_kernel(const uint32_t* __restrict__ tiles, int64_t n,
                                                                    uint32_t* __restrict__ ranges) {
  chain_begin();
  tile_ranges_body(tiles, n, ranges);
}

// Launches a pass kernel (its shared memory limit raised on its first use on a device).
template <typename S, typename... P, typename... A>
static Status launch_pass(Ctx* c, void (*kernel)(P...), size_t smem, uint64_t tiles, A... args) {
  static std::mutex guard;
  static std::set<std::pair<int, const void*>> ready;
  {
    std::lock_guard<std::mutex> lock(guard);
    const std::pair<int, const void*> key(c->device, reinterpret_cast<const void*>(kernel));
    if (!ready.count(key)) {
      SPLAT_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      ready.insert(key);
    }
  }
  return launch_chained(c, "radix_onesweep_kernel", kernel, (uint32_t)tiles, S::kThreads, smem, args...);
}

// SPLAT_PASS with the tile shape of a sort of `keys` (sort_tiles); 64-bit look-back words only
// come with more keys than the smaller shapes take.
#define SPLAT_PASS_BY_SIZE(keys)       \
  if constexpr (sizeof(W) == 8) {      \
    SPLAT_PASS(SortLarge);             \
  } else if (keys <= kSmallSortKeys) { \
    SPLAT_PASS(SortSmall);             \
  } else if (keys <= kMidSortKeys) {   \
    SPLAT_PASS(SortMid);               \
  } else {                             \
    SPLAT_PASS(SortLarge);             \
  }

template <bool kPacked, typename W>
static Status sort_entries(Ctx* c, const float* proj, const uint32_t* entry_offset, int64_t n, const KeyLayout& lay,
                           const uint32_t* depth_range, uint32_t depth_min, uint32_t tiles_x, const SortBuffers& buf,
                           uint32_t* gauss_out, uint64_t* keys_out, uint32_t* ranges) {
  const int64_t E = lay.E;
  uint64_t *ka = buf.ka, *kb = buf.kb;
  uint32_t *va = buf.va, *vb = buf.vb;
  const SortCtl ctl = carve_sort_ctl(buf.ctl, E);
  SPLAT_TRY(launch_chained(c, "emit_keys_kernel", emit_keys_kernel<kPacked>, emit_blocks(c, n), 256, 0,
                           reinterpret_cast<const float4*>(proj), entry_offset, n, tiles_x, depth_range, lay, ka, va,
                           ctl.hist));
  uint32_t* err = reinterpret_cast<uint32_t*>(static_cast<char*>(c->host_small_dev) + kAsyncErrorWordOffset);
  for (int p = 0; p < lay.passes; p++) {
    PassOut out{};
    out.last = p == lay.passes - 1;
    out.keys = kb;
    out.vals = out.last ? gauss_out : vb;
    out.tiles = reinterpret_cast<uint32_t*>(kb);  // the last pass leaves the key buffer free
    out.ref_keys = keys_out;
    out.depth_min = depth_min;
    out.vbits = lay.vbits;
    out.dbits = lay.dbits;
#define SPLAT_PASS(S)                                                                                          \
  SPLAT_TRY((launch_pass<S>(c, radix_onesweep_kernel<S, kPacked, W>, onesweep_smem<S, kPacked>(), sort_tiles(E), \
                            ka, va, E, p, ctl, err, out)))
    SPLAT_PASS_BY_SIZE(E)
#undef SPLAT_PASS
    std::swap(ka, kb);
    std::swap(va, vb);
  }
  SPLAT_TRY(launch_chained(c, "tile_ranges_kernel", tile_ranges_kernel, ceil_div(E, 4 * kRangeThreads),
                           kRangeThreads, 0, reinterpret_cast<const uint32_t*>(ka), E, ranges));
  return Status::ok();
}

Status launch_bin_sort_begin(Ctx* c, int64_t n, int64_t E, uint32_t width, uint32_t height, uint32_t* ranges,
                             const uint32_t* show, SortBuffers* buf) {
  const uint32_t num_tiles = c->raster.tiles(width, height);
  if (E == 0) return launch_zero3_u32(c, ranges, (size_t)num_tiles * 2, nullptr, 0, nullptr, 0, show);
  const int tbits = bits_for(num_tiles);
  SPLAT_TRY(arena_reserve(c, (size_t)E * 8, (void**)&buf->ka));
  SPLAT_TRY(arena_reserve(c, (size_t)E * 8, (void**)&buf->kb));
  if (tbits + 32 + bits_for((uint64_t)n) > 64) {  // keys may turn out too wide to pack
    SPLAT_TRY(arena_reserve(c, (size_t)E * 4, (void**)&buf->va));
    SPLAT_TRY(arena_reserve(c, (size_t)E * 4, (void**)&buf->vb));
  }
  SPLAT_TRY(arena_reserve(c, sort_ctl_bytes(E), &buf->ctl));
  const SortCtl ctl = carve_sort_ctl(buf->ctl, E);
  return launch_zero3_u32(c, ranges, (size_t)num_tiles * 2, ctl.status, status_bytes(E, max_passes(tbits)) / 4,
                          ctl.hist, kSortCounterWords, show);
}

Status launch_bin_sort(Ctx* c, const float* proj, const uint32_t* entry_offset, int64_t n, int64_t E,
                       const uint32_t* depth_range_dev, uint32_t depth_min, uint32_t depth_max, uint32_t width,
                       uint32_t height, const SortBuffers& buf, uint32_t* gauss_out, uint64_t* keys_out,
                       uint32_t* ranges) {
  if (E == 0) return Status::ok();
  const uint32_t tiles_x = c->raster.tiles_x(width), num_tiles = c->raster.tiles(width, height);
  const int tbits = bits_for(num_tiles), nbits = bits_for((uint64_t)n);
  KeyLayout lay;
  lay.E = E;
  lay.dbits = bits_for((uint64_t)(depth_max - depth_min) + 1);
  lay.passes = std::max(1, (tbits + lay.dbits + 7) / 8);
  const bool packed = tbits + lay.dbits + nbits <= 64;
  lay.vbits = packed ? nbits : 0;
#define SPLAT_SORT(P, W)                                                                                      \
  sort_entries<P, W>(c, proj, entry_offset, n, lay, depth_range_dev, depth_min, tiles_x, buf, gauss_out, keys_out, \
                     ranges)
  if (wide_words(E)) return packed ? SPLAT_SORT(true, uint64_t) : SPLAT_SORT(false, uint64_t);
  return packed ? SPLAT_SORT(true, uint32_t) : SPLAT_SORT(false, uint32_t);
#undef SPLAT_SORT
}

// ---------------------------------------------------------------------------------------
// Device-driven binning: the entry count and the depth range stay in device memory, so the
// host never waits for them. Grids and buffers are sized for a capacity E_cap; every
// kernel reads the count (clamped to E_cap) and the key width from device memory, skips
// passes the keys do not need, and the last needed pass writes the caller's buffer. An
// entry count above E_cap sets *overflow (sticky) and sorts only the first E_cap entries;
// the caller must discard that view's results. Keys and passes are launch_bin_sort's (packed
// when tile, Gaussian and 32 depth bits fit), so the output
// equals it.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ KeyLayout dev_layout(const uint64_t* __restrict__ E_dev, int64_t E_cap,
                                                const uint32_t* __restrict__ dr, int tbits, int vbits) {
  KeyLayout p;
  const uint64_t e = *E_dev;
  p.E = e < (uint64_t)E_cap ? (int64_t)e : E_cap;
  const uint32_t span = p.E > 0 ? dr[1] - dr[0] : 0u;
  p.dbits = span == 0 ? 0 : 32 - __clz(span);
  p.vbits = vbits;
  const int total = p.dbits + tbits;
  p.passes = total == 0 ? 1 : (total + 7) / 8;
  return p;
}

template <bool kPacked>
__global__ void __launch_bounds__(256) emit_keys_dev_kernel(
    const float4* __restrict__ rec, const uint32_t* __restrict__ entry_offset, int64_t n, uint32_t tiles_x,
    const uint32_t* __restrict__ depth_range, const uint64_t* __restrict__ E_dev, int64_t E_cap, int tbits, int vbits,
    uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t* __restrict__ hist,
    uint32_t* __restrict__ overflow, const BatchTable* __restrict__ bt, int64_t n_view) {
  chain_begin();
  const KeyLayout lay = dev_layout(E_dev, E_cap, depth_range, tbits, vbits);
  if (blockIdx.x == 0 && threadIdx.x == 0 && *E_dev > (uint64_t)E_cap) atomicOr(overflow, 1u);
  emit_keys_body<kPacked>(rec, entry_offset, n, tiles_x, depth_range, lay, E_cap, keys, vals, hist, bt, n_view);
}

struct DevBuffers {
  uint64_t *ka, *kb;
  uint32_t *va, *vb;
};

template <typename S, bool kPacked, typename W>
__global__ void __launch_bounds__(S::kThreads) radix_onesweep_dev_kernel(
    DevBuffers b, const uint64_t* __restrict__ E_dev, int64_t E_cap, const uint32_t* __restrict__ dr, int tbits,
    int vbits, int pass, SortCtl ctl, uint64_t tiles_cap, uint32_t* __restrict__ err, uint32_t* __restrict__ vals_final) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char dsm[];
  const KeyLayout lay = dev_layout(E_dev, E_cap, dr, tbits, vbits);
  if (pass >= lay.passes) return;
  const bool odd = pass & 1;
  PassOut out{};
  out.last = pass == lay.passes - 1;
  out.keys = odd ? b.ka : b.kb;
  out.vals = out.last ? vals_final : (odd ? b.va : b.vb);
  out.tiles = reinterpret_cast<uint32_t*>(out.keys);
  out.vbits = lay.vbits;
  out.dbits = lay.dbits;
  onesweep_body<S, kPacked, W>(odd ? b.kb : b.ka, odd ? b.vb : b.va, lay.E, 8 * pass + lay.vbits, ctl.hist + 256 * pass,
                               static_cast<W*>(ctl.status) + (size_t)pass * tiles_cap * 256, ctl.ticket + pass,
                               ctl.abort, err, out, dsm);
}

__global__ void __launch_bounds__(kRangeThreads) tile_ranges_dev_kernel(DevBuffers b, const uint64_t* __restrict__ E_dev,
                                                                        int64_t E_cap, const uint32_t* __restrict__ dr,
                                                                        int tbits, uint32_t* __restrict__ ranges) {
  chain_begin();
  const KeyLayout lay = dev_layout(E_dev, E_cap, dr, tbits, 0);
  // The tiles are where the last pass would have written keys.
  tile_ranges_body(reinterpret_cast<const uint32_t*>((lay.passes - 1) & 1 ? b.ka : b.kb), lay.E, ranges);
}

// Never less for a larger capacity, so that scratch for one serves every smaller one: the look-back
// words shrink where larger tiles come in (65,536 keys take 64 tiles of 1,024, 65,537 take 33 of
// 2,048), so a size covers the largest sort of each smaller shape too.
size_t dev_sort_scratch_bytes(int64_t E_cap) {
  const int64_t cap = std::max<int64_t>(E_cap, 1);
  size_t ctl = sort_ctl_bytes(cap);
  for (const int64_t last : {kSmallSortKeys, kMidSortKeys}) ctl = std::max(ctl, sort_ctl_bytes(std::min(cap, last)));
  return (size_t)cap * 24 + ctl + 6 * 256;  // 5 pieces, 256-aligned wherever the scratch starts
}

template <bool kPacked, typename W>
static Status sort_entries_dev(Ctx* c, const float* proj, const uint32_t* entry_offset, int64_t n,
                               const uint64_t* E_dev, int64_t E_cap, const uint32_t* dr, uint32_t tiles_x,
                               uint32_t num_tiles, int tbits, int vbits, void* scratch, uint32_t* gauss_out,
                               uint32_t* ranges, uint32_t* overflow, const BatchTable* bt, int64_t n_view) {
  const int64_t cap = std::max<int64_t>(E_cap, 1);
  const uint64_t tiles = sort_tiles(cap);
  // Carve the scratch (256-byte aligned pieces: the caller's base may have any alignment, and the
  // range kernel reads 16 bytes at a time).
  scratch = reinterpret_cast<void*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~(uintptr_t)255);
  auto carve = [&](size_t bytes) {
    void* p = scratch;
    scratch = static_cast<char*>(scratch) + ((bytes + 255) & ~(size_t)255);
    return p;
  };
  DevBuffers b;
  b.ka = static_cast<uint64_t*>(carve((size_t)cap * 8));
  b.kb = static_cast<uint64_t*>(carve((size_t)cap * 8));
  b.va = static_cast<uint32_t*>(carve((size_t)cap * 4));
  b.vb = static_cast<uint32_t*>(carve((size_t)cap * 4));
  const SortCtl ctl = carve_sort_ctl(carve(sort_ctl_bytes(cap)), cap);
  // One launch clears the tile ranges, the look-back words of the passes these keys can need,
  // and the histograms, tickets and abort word.
  SPLAT_TRY(launch_zero3_u32(c, ranges, (size_t)num_tiles * 2, ctl.status, status_bytes(cap, max_passes(tbits)) / 4, ctl.hist,
                             kSortCounterWords));
  if (n > 0) {
    SPLAT_TRY(launch_chained(c, "emit_keys_dev_kernel", emit_keys_dev_kernel<kPacked>, emit_blocks(c, n), 256, 0,
                             reinterpret_cast<const float4*>(proj), entry_offset, n, tiles_x, dr, E_dev, E_cap,
                             tbits, vbits, b.ka, b.va, ctl.hist, overflow, bt, n_view));
  }
  for (int pass = 0; pass < max_passes(tbits); pass++) {
#define SPLAT_PASS(S)                                                                                          \
  SPLAT_TRY((launch_pass<S>(c, radix_onesweep_dev_kernel<S, kPacked, W>, onesweep_smem<S, kPacked>(), tiles, b, \
                            E_dev, E_cap, dr, tbits, vbits, pass, ctl, tiles, overflow, gauss_out)))
    SPLAT_PASS_BY_SIZE(cap)
#undef SPLAT_PASS
  }
  SPLAT_TRY(launch_chained(c, "tile_ranges_dev_kernel", tile_ranges_dev_kernel, ceil_div(cap, 4 * kRangeThreads),
                           kRangeThreads, 0, b, E_dev, E_cap, dr, tbits, ranges));
  return Status::ok();
}

Status launch_bin_sort_dev(Ctx* c, const float* proj, const uint32_t* entry_offset, int64_t n, const uint64_t* E_dev,
                           int64_t E_cap, const uint32_t* depth_range_dev, uint32_t width, uint32_t height,
                           void* scratch, uint32_t* gauss_out, uint32_t* ranges, uint32_t* overflow,
                           const BatchTable* bt, int64_t n_view, uint32_t tiles_cap) {
  const uint32_t tiles_x = c->raster.tiles_x(width), tiles_y = c->raster.tiles_y(height);
  const uint32_t num_tiles = bt ? tiles_cap : tiles_x * tiles_y;
  const int tbits = bits_for(num_tiles), nbits = bits_for((uint64_t)std::max<int64_t>(n, 1));
  const bool packed = tbits + 32 + nbits <= 64;
  const int vbits = packed ? nbits : 0;
  n_view = std::max<int64_t>(n_view, 1);
#define SPLAT_SORT(P, W)                                                                                              \
  sort_entries_dev<P, W>(c, proj, entry_offset, n, E_dev, E_cap, depth_range_dev, tiles_x, num_tiles, tbits, vbits, \
                         scratch, gauss_out, ranges, overflow, bt, n_view)
  if (wide_words(E_cap)) return packed ? SPLAT_SORT(true, uint64_t) : SPLAT_SORT(false, uint64_t);
  return packed ? SPLAT_SORT(true, uint32_t) : SPLAT_SORT(false, uint32_t);
#undef SPLAT_SORT
}

#undef SPLAT_PASS_BY_SIZE

}  // namespace splat
