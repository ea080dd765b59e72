"""The binomial draws decided in FP32 (dust2gpu/binomial_filter.hpp) against
the FP64 samplers: the same integer, the same generator state afterwards,
for counts from 1 to 2^24 - 1 and means over the whole range of both
samplers and their boundary at n p = 10.  On the host every
special-function result is moved by its documented error bound, up or
down at random; on the device the real units are used.

Undecided draws are expected near one in 10^3 over this mix of counts
(the mean band is about 1e-3 of the unit spacing at the largest counts);
more than one in 100 would mean the bounds have become useless."""
import pathlib
import shutil
import subprocess

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent
SRC = ROOT / "tests" / "binomial_filter_check.cu"
CSRC = ROOT / "dust2_gb300" / "csrc"


def run(exe, *args):
    res = subprocess.run([str(exe), *map(str, args)], capture_output=True,
                         text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    draws, undecided, wrong = map(int, res.stdout.split())
    assert wrong == 0
    assert undecided < draws / 100
    return draws


@pytest.mark.parametrize("seed", [1, 2])
def test_decided_draws_equal_fp64_on_host(tmp_path, seed):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "filter_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(CSRC), "-x", "c++", str(SRC), "-o", str(exe)],
                   check=True)
    assert run(exe, 60000, 100, seed) > 6000000


@pytest.mark.gpu
def test_decided_draws_equal_fp64_on_device(built, tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "filter_check"
    subprocess.run([nvcc, "-O3", "-std=c++17", "-fmad=false", "-gencode",
                    "arch=compute_103a,code=sm_103a", "-I", str(CSRC),
                    str(SRC), "-o", str(exe)], check=True)
    assert run(exe, 32, 64) == 32 * 128 * 64 * 64
