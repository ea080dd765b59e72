"""Gradients by a group of lanes per particle, and by a thread per particle
(engine/unfilter.cuh): particle counts either side of the choice, time
steps that make the last tape shorter than a group, data every few steps,
resets between data times, and saved trajectories.  Exact, as the adjoint
tests are: every path sums the same values in the same order."""

import numpy as np
import pytest

import dust2_gb300 as d

pytestmark = pytest.mark.gpu


def pars_of(n):
    rs = np.random.default_rng(n)
    return [{"beta": rs.uniform(0.1, 0.5), "gamma": rs.uniform(0.05, 0.3),
             "N": float(rs.integers(500, 5000)), "I0": 10.0,
             "exp_noise": 1e6} for _ in range(n)]


@pytest.mark.parametrize("n_groups,n_times,every,dt", [
    (1, 1, 1, 1), (1, 33, 3, 0.5), (31, 40, 1, 1), (609, 9, 2, 0.25),
    (700, 33, 1, 1), (7400, 5, 1, 1)])
def test_gradient_matches_oracle(port, n_groups, n_times, every, dt):
    gen = d.sir()
    times = every * np.arange(1.0, n_times + 1)
    rs = np.random.default_rng(3)
    inc = rs.poisson(20, (n_times, n_groups)).astype(float)
    data = {"time": np.repeat(times, n_groups), "incidence": inc.ravel()}
    pars = pars_of(n_groups)
    if n_groups > 1:
        data["group"] = np.tile(np.arange(1, n_groups + 1), n_times)
    obj = d.dust_unfilter_create(gen, 0, data, dt=dt)
    ll = d.dust_likelihood_run(obj, pars if n_groups > 1 else pars[0],
                               adjoint=True, save_trajectories=True)
    gr = d.dust_likelihood_last_gradient(obj)
    flat = np.concatenate([gen.pack_pars(p) for p in pars])
    want_ll, want_gr, _ = port.unfilter_adjoint(
        "sir", flat, n_groups, 1, 0.0, times, inc.ravel(), n_groups, 5,
        dt=dt)
    np.testing.assert_array_equal(np.ravel(ll), np.ravel(want_ll))
    np.testing.assert_array_equal(np.reshape(gr, (3, n_groups)),
                                  want_gr.reshape(n_groups, 3).T)
    tr = d.dust_likelihood_last_trajectories(obj)
    plain = d.dust_unfilter_create(gen, 0, data, dt=dt)
    d.dust_likelihood_run(plain, pars if n_groups > 1 else pars[0],
                          adjoint=False, save_trajectories=True)
    np.testing.assert_array_equal(
        tr, d.dust_likelihood_last_trajectories(plain))
