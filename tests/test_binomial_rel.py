"""Binomial draws whose probability is known to a bound only
(dust2gpu/binomial_filter.hpp, `rel`): decided draws and SEIR steps on
counts equal the FP64 sampler's and update()'s, whatever the bound is.

More than one undecided draw in 1000 at bounds of 2^-24 and below (those of
ordinary tables) would mean that the bounds have become useless there."""
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path_factory.mktemp("rel") / "rel_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "dust2_gb300" / "csrc"),
                    str(ROOT / "tests" / "binomial_rel_check.cpp"), "-o",
                    str(exe)], check=True)

    def run(*args):
        res = subprocess.run([str(exe), *map(str, args)],
                             capture_output=True, text=True, timeout=300)
        assert res.returncode == 0, res.stdout + res.stderr
        return map(int, res.stdout.split())
    return run


@pytest.mark.parametrize("seed", [1, 2])
def test_decided_draws_with_inexact_probability(check, seed):
    draws, undecided, wrong = check("draws", 300000, seed)
    assert draws == 14 * 300000
    assert wrong == 0
    assert undecided < draws / 1000


@pytest.mark.parametrize("seed", [1, 2])
def test_seir_steps_with_coarse_coefficients(check, seed):
    steps, _, wrong = check("seir", 40000, seed)
    assert steps == 12 * 40000
    assert wrong == 0


@pytest.mark.gpu
@pytest.mark.parametrize("spread", [3, 7])
def test_seir_on_device_with_wide_contacts(port, spread):
    """Contacts over `spread` orders of magnitude, infected in one age at
    first: state and generators as the oracle's."""
    import dust2_gb300 as d
    gen = d.seir_age()
    rs = np.random.default_rng(spread)
    pars = {"R0": 2.5, "sigma": 0.5, "gamma": 0.2, "size": 20, "I0": 0,
            "N": np.full(16, 2e6),
            "contact": 10.0 ** rs.uniform(-spread, 0, 256)}
    n, dt = 333, 0.25
    start = np.zeros((96, n))
    start[0:16] = 2e6
    start[0] -= 3e5
    start[32] = 3e5
    sys = d.dust_system_create(gen, pars, n_particles=n, dt=dt, seed=8)
    words = np.frombuffer(d.dust_system_rng_state(sys), dtype="<u8")
    d.dust_system_set_state(sys, start)
    d.dust_system_run_to_time(sys, 12)
    got = d.dust_system_state(sys)
    out, rng_out = port.discrete_simulate(
        "seir_age", gen.pack_pars(pars), 1, n, 0.0, dt, words, [12.0],
        initial=np.ascontiguousarray(start.T.ravel()))
    np.testing.assert_array_equal(got.T.ravel(), out[:got.size])
    rng = np.frombuffer(d.dust_system_rng_state(sys), dtype="<u8")
    np.testing.assert_array_equal(rng, rng_out)
