"""The mixed-time filter with between two and three warps of particles per SM
partition (45,000 particles here; engine/filter.cuh k_step_compare_mixed)
against fewer (12,000): with no data a particle's path depends on its own
stream only, the first particles have the same streams, and the two kernels
are one source, so the states are the same bits.  One group, and two whose
last tiles have a remainder."""

import numpy as np
import pytest

import dust2_gb300 as d

pytestmark = pytest.mark.gpu


def final_state(n_groups, n_particles, n_rates):
    times = np.array([1.0, 3, 4])
    data = {"time": np.repeat(times, n_groups),
            "tested": np.full(3 * n_groups, 50.0),
            "positive": np.full(3 * n_groups, np.nan)}
    if n_groups > 1:
        data["group"] = np.tile(np.arange(1, n_groups + 1), 3)
    obj = d.dust_filter_create(d.malaria(), 0, data, dt=0.5, seed=4,
                               n_particles=n_particles)
    pars = {"n_rates": n_rates, "a": 0.3}
    d.dust_likelihood_run(obj, [pars] * n_groups if n_groups > 1 else pars)
    state = d.dust_likelihood_last_state(obj)
    return state[..., 0] if n_groups > 1 else state


@pytest.mark.parametrize("n_rates", [1, 15, 19])
@pytest.mark.parametrize("n_groups,many,few", [(1, 45000, 12000),
                                               (2, 22517, 6001)])
def test_three_warps_match_two(built, n_rates, n_groups, many, few):
    got = final_state(n_groups, many, n_rates)
    want = final_state(n_groups, few, n_rates)
    assert want.shape == (n_rates + 5, few)
    np.testing.assert_array_equal(got[:, :few], want)
