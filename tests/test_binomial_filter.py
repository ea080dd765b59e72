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


@pytest.mark.parametrize("seed", [1, 2])
def test_count_update_equals_update(tmp_path, seed):
    """Count stepping of sir, sir_cases and seir_age against their
    update(): hazards from 2^-30 a person to above 1/2, flipped and zero
    probabilities, populations up to 2^24, ages without infected, contact
    entries over five orders of magnitude.  About one case in ten is
    outside what the tables hold (a rate of 0, say) and is not counted."""
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "count_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(CSRC), str(ROOT / "tests" / "count_update_check.cpp"),
                    "-o", str(exe)], check=True)
    res = subprocess.run([str(exe), "6000", str(seed)], capture_output=True,
                         text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    steps, wrong, unfit = map(int, res.stdout.split())
    assert wrong == 0
    assert steps > 60 * 6000 and unfit < 6000 / 5


@pytest.mark.gpu
@pytest.mark.parametrize("n_pop,i0,beta,dt", [
    (1000, 10, 0.4, 0.25),        # counts, small probabilities
    (16777000, 5000, 2.5, 1),     # near the FP32 limit, hazards above 1/2
    (20000000, 100, 0.5, 0.25),   # beyond it: update()
    (1000.5, 10, 0.4, 0.25),      # not counts: update()
    (500, 10, 0, 0.25),           # no infection: update()
])
def test_count_stepping_on_device(port, n_pop, i0, beta, dt):
    """Stepping on the device, whichever way a particle takes, against the
    oracle: state and generators exactly."""
    import numpy as np

    import dust2_gb300 as d
    gen = d.sir_cases()
    pars = {"N": n_pop, "I0": i0, "beta": beta, "gamma": 0.3}
    sys = d.dust_system_create(gen, pars, n_particles=333, dt=dt, seed=3)
    words = np.frombuffer(d.dust_system_rng_state(sys), dtype="<u8")
    d.dust_system_set_state_initial(sys)
    d.dust_system_run_to_time(sys, 40)
    got = d.dust_system_state(sys)
    out, rng_out = port.discrete_simulate("sir_cases", gen.pack_pars(pars),
                                          1, 333, 0.0, dt, words, [40.0])
    np.testing.assert_array_equal(got.T.ravel(), out[:got.size])
    rng = np.frombuffer(d.dust_system_rng_state(sys), dtype="<u8")
    np.testing.assert_array_equal(rng, rng_out)
