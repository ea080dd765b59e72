"""Resampled particles moved by the step that follows (it reads the state of
its ancestor) against moving them after each resampling, which a run that
saves trajectories does.  Exact: the same particles either way.  With data
missing at some times (nothing is resampled), a time at which every density
is -Inf (all follow the first particle), every kind of step launch, and runs
of some of the groups."""

import numpy as np
import pytest

import dust2_gb300 as d
from dust2_gb300 import interface
from test_gpu_filter import _uneven_case
from test_gpu_simulate import _pars

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n_particles,shape", [
    ("sir_cases", [257, 40, 1, 600], None),
    ("sir_cases", [257, 40, 1, 600], (32, 3, False)),
    ("sir_cases", [5000, 4097], (256, 0, True)),
    ("sirs", [130, 70], (64, 0, False)),
    ("seir_age", [33, 161, 70], None),
    ("seir_age", [33, 161, 70], (128, 0, True))])
def test_moved_by_step_is_identical(built, name, n_particles, shape):
    gen = d.Generator(name)
    G = len(n_particles)
    _, times, data = _uneven_case(5, n_particles, n_times=11)
    data[4] = np.nan
    data[6, 0] = 1e307
    cols = {"time": np.repeat(times, G), "group": np.tile(np.arange(1, G + 1),
                                                          times.size),
            gen.data_names[0]: data.ravel()}
    pars = _pars(name, G)
    out = []
    for history in (False, True):
        obj = d.dust_filter_create(gen, 0, cols, n_particles=n_particles,
                                   dt=0.25, seed=11)
        interface.dust_likelihood_set_fused_tail(obj, False)
        if shape is not None:
            interface.dust_likelihood_set_step_shape(obj, *shape)
        res = []
        for groups in (None, [G], None, [2, 1]):
            p = pars if groups is None else [pars[i - 1] for i in groups]
            res.append(d.dust_likelihood_run(obj, p, index_group=groups,
                                             save_trajectories=history))
            # the state of the groups that were run comes first
            n = obj.n_state * sum(n_particles[i - 1] for i in
                                           groups or range(1, G + 1))
            res.append(d.dust_likelihood_last_state(obj)[:n])
        res.append(np.frombuffer(d.dust_likelihood_rng_state(obj), "<u8"))
        out.append(res)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
