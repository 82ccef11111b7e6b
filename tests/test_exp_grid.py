"""The compositing forward's exp (crmath.h: expf_cr_grid, its table built at compile time)
equals the general correctly rounded exp on its range. The header is plain C++ on the host,
with the same double operations as on the device."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include <cstdio>
#include <cstring>
#include "crmath.h"
static constexpr crm::ExpGrid G;
static long check(unsigned lo, unsigned hi, unsigned step) {
  long bad = 0;
  for (unsigned long u = lo; u <= hi; u += step) {
    const unsigned b = (unsigned)u;
    float s;
    std::memcpy(&s, &b, 4);
    const float want = crm::expf_cr(-s), got = crm::expf_cr_grid(s, G.v);
    bad += std::memcmp(&want, &got, 4) != 0;
  }
  return bad;
}
int main() {
  unsigned top, low;
  const float max = crm::kExpGridMax, one = 0.0009765625f;
  std::memcpy(&top, &max, 4);
  std::memcpy(&low, &one, 4);
  long bad = check(0, low, 4099) + check(low, top, 53) + check(top - 100000, top, 1);
  const float zero = crm::expf_cr_grid(crm::kExpGridSkip, G.v);
  std::printf("%ld %d\n", bad, zero == 0.0f);
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_exp_grid_equals_the_correctly_rounded_exp(tmp_path):
    src, exe = tmp_path / "grid.cpp", tmp_path / "grid"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-mfma",
                    "-I" + os.path.join(ROOT, "splatrs_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300).stdout.split()
    assert out == ["0", "1"]
