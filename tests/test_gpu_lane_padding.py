"""The mixed-time filter with a particle's variables over lanes, where the
lanes' last entries are padding: with an absolute tolerance of 0 (which the
C ABI accepts) padding has no error scale, and must not count.  Against a
thread per particle, which has no padding (12,000 particles), as
test_gpu_mixed_lanes.py does and with its tolerance."""

import numpy as np
import pytest

import dust2_gb300 as d

pytestmark = pytest.mark.gpu


def final_state(n_particles, n_rates, initial):
    times = np.array([1.0, 3, 4, 6])
    data = {"time": times, "tested": np.array([50.0, np.nan, 80, 20]),
            "positive": np.full(4, np.nan)}
    control = dict(d.dust_ode_control(), atol=0.0)
    obj = d.dust_filter_create(d.malaria(), 0, data, dt=1, seed=4,
                               n_particles=n_particles, ode_control=control)
    d.dust_likelihood_run(obj, {"n_rates": n_rates, "a": 0.3},
                          initial=np.repeat(initial[:, None], n_particles,
                                            axis=1))
    return d.dust_likelihood_last_state(obj)


@pytest.mark.parametrize("n_rates", [1, 7, 15, 19])
def test_no_absolute_tolerance(built, n_rates):
    initial = np.concatenate([[0.8, 0.2, 0.9, 0.05],
                              np.full(n_rates, 0.05 / n_rates), [0.1]])
    few = final_state(33, n_rates, initial)
    many = final_state(12000, n_rates, initial)
    assert np.all(np.isfinite(few))
    np.testing.assert_allclose(few, many[:, :33], rtol=1e-9, atol=1e-12)
