"""The mixed-time filter with a particle's variables shared out over lanes
(few particles) against a thread per particle (more than 12 particles per SM
partition, so also 12,000 particles): the smallest, the largest and two
middle numbers of variables, an interval of several updates, and particle
counts that leave a tile part empty.  With no data a particle's path depends
on its own stream only, and the first particles of both filters have the
same streams.  (The golden fixtures of the mixed-time tests cover weights and
resampling with lanes.)

Tolerance 1e-9 relative, as the mixed-time tests have it: the error norm is
summed in another order."""

import numpy as np
import pytest

import dust2_gb300 as d

pytestmark = pytest.mark.gpu


def final_state(n_particles, n_rates, dt, tested):
    times = np.array([1.0, 3, 4, 6])
    data = {"time": times, "tested": tested,
            "positive": np.full(4, np.nan)}
    obj = d.dust_filter_create(d.malaria(), 0, data, dt=dt, seed=4,
                               n_particles=n_particles)
    pars = {"n_rates": n_rates, "a": 0.3}
    out = []
    for _ in range(2):
        d.dust_likelihood_run(obj, pars)
        out.append(d.dust_likelihood_last_state(obj))
    return out


@pytest.mark.parametrize("n_rates,n_particles,dt", [
    (1, 1, 1), (7, 33, 0.5), (15, 101, 1), (19, 250, 0.25)])
def test_lanes_match_threads(built, n_rates, n_particles, dt):
    tested = np.array([50.0, np.nan, 80, 20])
    few = final_state(n_particles, n_rates, dt, tested)
    many = final_state(12000, n_rates, dt, tested)
    for a, b in zip(few, many):
        assert a.shape == (n_rates + 5, n_particles)
        np.testing.assert_allclose(a, b[:, :n_particles], rtol=1e-9,
                                   atol=1e-12)
