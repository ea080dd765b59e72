"""The one-launch tail for groups above 1024 particles: one particle more
than the small cluster holds, an odd number, and the most the large one
holds, against the separate kernels.  Exact: both form the same sums in the
same structure."""

import numpy as np
import pytest

import dust2_gb300 as d
from dust2_gb300 import interface
from test_gpu_filter import _uneven_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_particles", [[1025, 40, 2047], [3001], [4096] * 3])
def test_large_fused_tail_is_identical(built, n_particles):
    gen = d.sir_cases()
    plist, times, data = _uneven_case(5, n_particles, n_times=12)
    G = len(n_particles)
    data[3, 0] = 1e307  # a time at which every log density is -Inf
    cols = {"time": np.repeat(times, G), "incidence": data.ravel()}
    if G > 1:
        cols["group"] = np.tile(np.arange(1, G + 1), times.size)
    pars = plist if G > 1 else plist[0]
    for serial in (False, True):
        res = []
        for fused in (True, False):
            obj = d.dust_filter_create(gen, 0, cols, n_particles=n_particles,
                                       dt=0.25, seed=11)
            interface.dust_likelihood_set_fused_tail(obj, fused)
            interface.dust_likelihood_set_serial_resample(obj, serial)
            ll = [d.dust_likelihood_run(obj, pars) for _ in range(2)]
            res.append((np.array(ll), d.dust_likelihood_last_state(obj),
                        d.dust_likelihood_rng_state(obj),
                        d.dust_likelihood_serial_fallbacks(obj)))
        np.testing.assert_array_equal(res[0][0], res[1][0])
        np.testing.assert_array_equal(res[0][1], res[1][1])
        assert res[0][2] == res[1][2]
        assert res[0][3] == res[1][3]
        assert (res[0][3] > 0) == serial
