// Parameter planes to a host array of reference Gaussian records, for host memory that is neither
// pinned nor, often, mapped yet. The device converts and copies 44 MB in a millisecond; the rest of
// the 10 ms that a fresh array took was its pages' first touch, taken one by one under the driver's
// single-threaded copy. Here several threads touch them, while the device converts the records:
// 187k Gaussians 9.8-15.4 -> 6.7-11.7 ms by machine, and no slower the first time.
// (Pinned slots emptied by several threads were faster on a repeated call, 4.3 ms, but their
// allocation made a context's first call 3-20 ms longer.)
#include <algorithm>
#include <exception>
#include <thread>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "renderer.cuh"

namespace splat {

constexpr size_t kPage = 4096, kTouchPart = 1 << 20;
constexpr unsigned kMaxThreads = 8;

// One write access per page that changes nothing.
static void touch(char* a, char* end) {
  while (a < end) {
    __atomic_fetch_or(a, 0, __ATOMIC_RELAXED);
    a = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(a) & ~(uintptr_t)(kPage - 1)) + kPage);
  }
}

static void touch_pages(char* host, size_t bytes) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, host) != cudaSuccess) {
    cudaGetLastError();
    return;
  }
  if (at.type != cudaMemoryTypeUnregistered) return;  // pinned or managed: mapped already
  const unsigned threads = (unsigned)std::min<size_t>(
      bytes / kTouchPart, std::min(kMaxThreads, std::thread::hardware_concurrency() / 2));
  if (threads < 2) return;  // the copy touches a small array as fast
  const size_t part = bytes / threads;
  std::vector<std::thread> pool;
  try {
    pool.reserve(threads);
    for (unsigned t = 0; t < threads; t++)
      pool.emplace_back(touch, host + t * part, t + 1 == threads ? host + bytes : host + (t + 1) * part);
  } catch (const std::exception&) {
    // Fewer threads than wanted: the copy touches what they don't.
  }
  for (std::thread& t : pool) t.join();
}

Status download_records(Ctx* c, const float* planes, int64_t n, int64_t cap, float* aos_host) {
  const size_t bytes = (size_t)n * 59 * 4;
  DevBuf tmp;
  Status s = tmp.ensure(std::max<size_t>(bytes, 4));
  if (s.good()) s = launch_params_to_aos(c, planes, n, cap, tmp.as<float>());
  if (s.good() && n) {
    touch_pages(reinterpret_cast<char*>(aos_host), bytes);
    s = cuda_status(cudaMemcpyAsync(aos_host, tmp.ptr, bytes, cudaMemcpyDeviceToHost, c->stream), "download records");
  }
  if (s.good()) s = cuda_status(cudaStreamSynchronize(c->stream), "cudaStreamSynchronize");
  tmp.release();
  return s;
}

}  // namespace splat
