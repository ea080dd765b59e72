"""math::is_multiple (the test of a reset time) against std::fmod(t, p) == 0:
whole and fractional times on both sides of zero, random bit patterns, and
zeros, subnormals, infinities and NaN in either argument."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
CHECK = r"""
#include <cmath>
#include <cstdio>
#include "dust2gpu/math.hpp"
using namespace dust2gpu;
static std::uint64_t s = 88172645463325252ull;
static std::uint64_t next() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static long bad, hits;
static void check(double t, double p) {
  const bool want = std::fmod(t, p) == 0;
  bad += math::is_multiple(t, p) != want;
  hits += want;
}
int main() {
  const double periods[] = {1, 2, 7, 0.25, 0.1, 0.5, 4, 3, 1024, 1e-3, 0x1p-30,
                            0x1p60, 0x1p-1022, 0x1p-1074, 0x1p1023, -1, -0.5,
                            0.0, -0.0, math::infinity(), math::quiet_nan()};
  const double times[] = {0.0, -0.0, 0x1p-1074, 0x1p-1022, 0x1.8p-1022, 0x1p52,
                          0x1p53, 0x1.fffffffffffffp52, 0x1p1023, 1e300,
                          math::infinity(), math::quiet_nan()};
  for (double p : periods) {
    for (double t : times) { check(t, p); check(-t, p); }
    for (int i = -4000; i < 4000; ++i) {
      check(i * 0.25, p); check(i * 0.1, p); check(i * p, p);
      check(i * (p / 4), p);
    }
    for (int i = 0; i < 20000; ++i) {
      check(math::from_bits(next()), p);
      check(math::from_bits(next() & (~0ull << (next() % 53))), p);
    }
  }
  std::printf("%ld %d\n", bad, hits > 10000);
}
"""


def test_reset_times_are_those_of_fmod(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    src = tmp_path / "check.cpp"
    src.write_text(CHECK)
    exe = tmp_path / "check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "dust2_gb300" / "csrc"), str(src), "-o",
                    str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True,
                         timeout=300)
    assert res.stdout.split() == ["0", "1"]
