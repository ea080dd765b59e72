"""The kernels that run update() in FP64 (deterministic likelihoods and
gradients by threads) keep the registers they had before the count-stepping
kernels were compiled for more blocks per SM: with 64 instead of 128,
k_unfilter_adjoint<sir> spilled 204 bytes, and 4096 deterministic SEIR
particles took 39.2 ms instead of 33.7."""
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_blocks_per_sm(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "bounds"
    subprocess.run(
        [nvcc, "-std=c++17", "--expt-relaxed-constexpr", "-gencode",
         "arch=compute_103a,code=sm_103a", "-I",
         str(ROOT / "dust2_gb300" / "csrc"),
         str(ROOT / "tests" / "kernel_bounds.cu"), "-o", str(exe)],
        check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True,
                         check=True).stdout.split()
    #              sir       sir_cases  seir_age  walk
    assert out == ["4", "2", "4", "2", "5", "4", "2", "2"]
