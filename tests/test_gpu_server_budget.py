"""The likelihood server's device memory stays within its budget: particles,
observations and the sessions' own data (engine/served.cuh), with so many
sessions that their parameters and count tables take a good part of it."""
import shutil
import subprocess

import pytest

import dust2_gb300 as d
from conftest import ROOT

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system", ["sir_cases", "seir_age"])
def test_budget_holds_the_sessions_tables(built, tmp_path, system):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "sizes"
    subprocess.run(
        [nvcc, "-std=c++17", "--expt-relaxed-constexpr", f"-DSYSTEM={system}",
         "-gencode", "arch=compute_103a,code=sm_103a", "-I",
         str(ROOT / "dust2_gb300" / "csrc"),
         str(ROOT / "tests" / "served_sizes.cu"), "-o", str(exe)],
        check=True)
    per_session, per_obs, per_particle = map(int, subprocess.run(
        [str(exe)], capture_output=True, text=True, check=True)
        .stdout.split())
    budget, n_sessions = 4e7, 4096
    server = d.dust_likelihood_server(getattr(d, system)(),
                                      hbm_budget=budget,
                                      max_sessions=n_sessions)
    cap = server.capacity()
    server.free()
    used = (cap["n_particles"] * per_particle +
            cap["n_observations"] * per_obs + n_sessions * per_session)
    assert 0.9 * budget < used <= budget
