"""The mixed-time filter's lanes serve systems of the shape they are written
for: one special entry, no outputs, no resets.  Any other system is
integrated by a thread per particle, however few its particles."""
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_systems_served_by_lanes(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not shutil.which(nvcc):
        pytest.skip("nvcc not available")
    exe = tmp_path / "lanes"
    subprocess.run(
        [nvcc, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-gencode",
         "arch=compute_103a,code=sm_103a", "-I",
         str(ROOT / "dust2_gb300" / "csrc"),
         str(ROOT / "tests" / "lanes_contract.cu"), "-o", str(exe)],
        check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True,
                         check=True)
    #                      malaria, sirode; special 1, 0, 2; output; resets
    assert res.stdout.strip() == "10" "100" "0" "10"
