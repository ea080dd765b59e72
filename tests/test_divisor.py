"""Division by an invariant (math::divisor): the fused form that the device
uses gives the correctly rounded quotient, compared with the host's
division on 20 million pairs, with significands of long runs of ones or
zeros among them, and arguments outside its range."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
CHECK = r"""
#include <cstdio>
#include "dust2gpu/math.hpp"
using namespace dust2gpu;
static std::uint64_t s = 88172645463325252ull;
static std::uint64_t next() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static long bad;
static void check(double a, double b) {
  const double got = math::divide_fma(a, math::divisor::of(b));
  const double want = a / b;
  const bool nan = got != got && want != want;
  bad += !nan && !(got == want);
}
int main() {
  const std::uint64_t m = 0x000fffffffffffffull;
  for (long i = 0; i < 20000000; ++i) {
    std::uint64_t u = next(), v = next();
    const int eu = 1023 + static_cast<int>(next() % 200) - 100;
    const int ev = 1023 + static_cast<int>(next() % 100) - 50;
    if (i % 5 == 0) v |= 0x000ffffffffffff0ull;
    if (i % 7 == 0) u |= 0x000fffffffffff00ull;
    if (i % 11 == 0) v &= 0xfull;
    if (i % 13 == 0) u &= 0xffull;
    check(math::from_bits((u & m) | (std::uint64_t(eu) << 52)),
          math::from_bits((v & m) | (std::uint64_t(ev) << 52)));
  }
  const double e[] = {0.0, 1e-320, 1e-308, 1e-130, 1, 3, 1e130, 1e300,
                      math::infinity(), math::quiet_nan()};
  for (double a : e) for (double b : e) { check(a, b); check(-a, b); check(a, -b); }
  std::printf("%ld\n", bad);
}
"""


def test_divide_by_invariant_is_correctly_rounded(tmp_path):
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
    assert res.stdout.split() == ["0"]
