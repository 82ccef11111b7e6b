"""The compositing forward's exp (crmath.h: expf_cr_grid, its table built at compile time)
equals the general correctly rounded exp on its range: every float of it, by several threads
(about 25 s of processor time). The header is plain C++ on the host, with the same double
operations as on the device, and the forward calls the same function."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
#include "crmath.h"
static constexpr crm::ExpGrid G;
static long check(unsigned lo, unsigned hi) {
  long bad = 0;
  for (unsigned b = lo; b < hi; b++) {
    float s;
    std::memcpy(&s, &b, 4);
    const float want = crm::expf_cr(-s), got = crm::expf_cr_grid(s, G.v);
    bad += std::memcmp(&want, &got, 4) != 0;
  }
  return bad;
}
int main() {
  unsigned top;
  const float max = crm::kExpGridMax;
  std::memcpy(&top, &max, 4);
  const unsigned kPart = 1u << 22;
  std::atomic<unsigned> next(0);
  std::atomic<long> bad(0);
  std::vector<std::thread> pool;
  for (unsigned t = 0; t < std::clamp(std::thread::hardware_concurrency(), 1u, 64u); t++)
    pool.emplace_back([&] {
      for (unsigned lo; (lo = next.fetch_add(1) * kPart) <= top;) bad += check(lo, std::min(top + 1, lo + kPart));
    });
  for (std::thread& t : pool) t.join();
  const float zero = crm::expf_cr_grid(crm::kExpGridSkip, G.v);
  std::printf("%ld %d\n", bad.load(), zero == 0.0f);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_exp_grid_equals_the_correctly_rounded_exp(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma", "-pthread",
                    "-I" + os.path.join(ROOT, "splatrs_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    assert out == ["0", "1"]
