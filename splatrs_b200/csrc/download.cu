// Parameter planes to a host array of reference Gaussian records, for host memory that is neither
// pinned nor, often, mapped yet: a fresh array's first touch and the driver's single-threaded copy
// out of its bounce buffer made 44 MB take 10 ms, 180 times what the device needs. Here the records
// of kChunk Gaussians at a time are converted on the device, copied to one of kSlots pinned slots,
// and written to the caller's array by several threads (so its pages are mapped by all of them)
// while the next chunks arrive. The slots (7.7 MB pinned, 7.7 MB on the device) belong to the
// context and go with it.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace splat {

constexpr int kSlots = 4;
constexpr int64_t kChunk = 8192;
constexpr size_t kChunkBytes = (size_t)kChunk * 59 * 4;
constexpr unsigned kMaxThreads = 8;

struct Download {
  void* host = nullptr;  // kSlots chunks, pinned
  void* dev = nullptr;
  cudaEvent_t arrived[kSlots] = {};
};

void download_free(Ctx* c) {
  Download* d = c->download;
  c->download = nullptr;
  if (!d) return;
  for (cudaEvent_t e : d->arrived)
    if (e) cudaEventDestroy(e);
  if (d->host) cudaFreeHost(d->host);
  if (d->dev) cudaFree(d->dev);
  delete d;
}

static Status download_ready(Ctx* c) {
  if (c->download) return Status::ok();
  c->download = new (std::nothrow) Download();
  if (!c->download) return Status::make(SPLAT_ERR_CUDA, "host allocation failed");
  Download* d = c->download;
  bool ok = cudaHostAlloc(&d->host, kSlots * kChunkBytes, cudaHostAllocDefault) == cudaSuccess;
  ok = ok && cudaMalloc(&d->dev, kSlots * kChunkBytes) == cudaSuccess;
  for (cudaEvent_t& e : d->arrived) ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (ok) return Status::ok();
  cudaGetLastError();
  download_free(c);
  return Status::make(SPLAT_ERR_CUDA, "allocation of the download slots failed");
}

// Queues chunk k's conversion and copy.
static Status send_chunk(Ctx* c, const float* planes, int64_t n, int64_t cap, int64_t k) {
  Download* d = c->download;
  const int64_t i0 = k * kChunk, cnt = std::min(kChunk, n - i0);
  const size_t at = (size_t)(k % kSlots) * kChunkBytes;
  float* dev = reinterpret_cast<float*>(static_cast<char*>(d->dev) + at);
  SPLAT_TRY(launch_params_to_aos(c, planes + 4 * i0, cnt, cap, dev));
  SPLAT_CUDA(cudaMemcpyAsync(static_cast<char*>(d->host) + at, dev, (size_t)cnt * 59 * 4, cudaMemcpyDeviceToHost,
                             c->stream));
  SPLAT_CUDA(cudaEventRecord(d->arrived[k % kSlots], c->stream));
  return Status::ok();
}

Status download_records(Ctx* c, const float* planes, int64_t n, int64_t cap, float* aos_host) {
  if (n == 0) {
    SPLAT_CUDA(cudaStreamSynchronize(c->stream));
    return Status::ok();
  }
  SPLAT_TRY(download_ready(c));
  Download* d = c->download;
  const int64_t chunks = (n + kChunk - 1) / kChunk;
  for (int64_t k = 0; k < std::min<int64_t>(chunks, kSlots); k++) SPLAT_TRY(send_chunk(c, planes, n, cap, k));
  // Thread t of T writes the t-th part of every chunk; `arrived` chunks may be read, `written[s]`
  // counts the parts written out of slot s since the start.
  std::atomic<int64_t> arrived{0};
  std::atomic<int64_t> written[kSlots] = {};
  std::atomic<bool> stop{false};
  unsigned threads = 1;
  auto part = [&](int64_t k, unsigned t) {
    const size_t bytes = (size_t)std::min(kChunk, n - k * kChunk) * 59 * 4;
    const size_t a = bytes / 64 * t / threads * 64, b = t + 1 == threads ? bytes : bytes / 64 * (t + 1) / threads * 64;
    std::memcpy(reinterpret_cast<char*>(aos_host) + (size_t)k * kChunkBytes + a,
                static_cast<const char*>(d->host) + (size_t)(k % kSlots) * kChunkBytes + a, b - a);
    written[k % kSlots].fetch_add(1, std::memory_order_release);
  };
  std::vector<std::thread> pool;
  if (chunks > 1) {
    const unsigned want = std::max(1u, std::min(kMaxThreads, std::thread::hardware_concurrency() / 2));
    try {
      pool.reserve(want);
      for (unsigned t = 1; t < want; t++)
        pool.emplace_back([&, t] {
          for (int64_t k = 0; k < chunks; k++) {
            while (arrived.load(std::memory_order_acquire) <= k) {
              if (stop.load(std::memory_order_relaxed)) return;
              std::this_thread::yield();
            }
            part(k, t);
          }
        });
    } catch (const std::exception&) {
      // Fewer threads than wanted: those that run are the team.
    }
    threads = (unsigned)pool.size() + 1;  // read by the team only after the first release of `arrived`
  }
  Status s = Status::ok();
  for (int64_t k = 0; k < chunks && s.good(); k++) {
    s = cuda_status(cudaEventSynchronize(d->arrived[k % kSlots]), "download records");
    if (!s.good()) break;
    arrived.store(k + 1, std::memory_order_release);
    part(k, 0);
    // The slot of chunk k is free for chunk k + kSlots once every part of it is written.
    const int64_t uses = k / kSlots + 1;
    if (k + kSlots < chunks) {
      while (written[k % kSlots].load(std::memory_order_acquire) < uses * (int64_t)threads) std::this_thread::yield();
      s = send_chunk(c, planes, n, cap, k + kSlots);
    }
  }
  if (!s.good()) stop.store(true);
  for (std::thread& t : pool) t.join();
  if (!s.good()) cudaStreamSynchronize(c->stream);  // nothing may still write the slots
  return s;
}

}  // namespace splat
