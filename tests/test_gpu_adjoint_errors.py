"""An error that a comparison raises at one data time reaches the caller
whichever kernel runs the gradient: a thread per particle, or lanes that
each compare other data times (engine/unfilter.cuh)."""
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_errors_of_any_data_time_are_reported(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "adjoint_errors"
    subprocess.run(
        [nvcc, "-O2", "-std=c++17", "-fmad=false", "--expt-relaxed-constexpr",
         "-gencode", "arch=compute_103a,code=sm_103a", "-I",
         str(ROOT / "dust2_gb300" / "csrc"),
         str(ROOT / "tests" / "adjoint_error_check.cu"), "-o", str(exe)],
        check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True,
                         timeout=120)
    assert res.returncode == 0, res.stdout + res.stderr
    rows = [line.split() for line in res.stdout.splitlines()]
    assert len(rows) == 5 * 3 * 5
    for i in range(0, len(rows), 15):
        fail = int(rows[i][0])
        threads = rows[i:i + 5]
        for row in threads:  # the first failing data time, or none
            assert (int(row[2]) != 0) == (fail >= 0)
            assert float(row[3]) == (fail + 1 if fail >= 0 else 0)
        for lanes in (rows[i + 5:i + 10], rows[i + 10:i + 15]):
            assert [r[2:] for r in lanes] == [r[2:] for r in threads]
