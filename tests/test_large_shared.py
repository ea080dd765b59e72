"""Systems with large parameter tables: a block stages a group's parameters
in its 48 KB of static shared memory, and what the simulation kernel keeps
beside them must leave the room that the other kernels do."""
import re
import shutil
import subprocess

import pytest

from conftest import ROOT


# the largest table that k_run takes, the largest beside which the reset
# tests of all of a launch's output times fit, and one more than that
@pytest.mark.parametrize("doubles", [6125, 5613, 5614])
def test_simulation_kernel_fits_where_others_do(doubles):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("nvcc not available")
    res = subprocess.run(
        [nvcc, "-O2", "-std=c++17", "-fmad=false", "--expt-relaxed-constexpr",
         f"-DSHARED_DOUBLES={doubles}", "-gencode",
         "arch=compute_103a,code=sm_103a", "-Xptxas", "-v", "-I",
         str(ROOT / "dust2_gb300" / "csrc"), "-c",
         str(ROOT / "tests" / "large_shared.cu"), "-o", "/dev/null"],
        capture_output=True, text=True, check=True)
    used = dict(re.findall(r"entry function '\S*?(k_run|k_simulate)I.*?"
                           r"(\d+) bytes smem", res.stderr, re.S))
    assert set(used) == {"k_run", "k_simulate"}, res.stderr
    assert int(used["k_run"]) <= 49152
    assert int(used["k_simulate"]) <= 49152
