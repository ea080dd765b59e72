"""A simulation in one launch per 128 output times, against a run to each
time and its state: more times than one launch takes, more steps to a time
than have their resets tested ahead (64), times without a step, groups that
share a block, and entries of the state in another order.  Exact: the same
steps, whichever launch takes them."""

import numpy as np
import pytest

import dust2_gb300 as d
from test_gpu_compat import PARS as SIRS
from test_gpu_system import plist_from
from conftest import golden

pytestmark = pytest.mark.gpu

TIMES = np.concatenate([np.arange(0, 33, 0.25), [50.25, 50.5, 90]])


def _pars(name, n_groups):
    if name == "seir_age":
        g = golden("simulate_seir_age")
        one = plist_from(d.Generator(name), g["pars"], int(g["n_groups"]))
        return (one * n_groups)[:n_groups]
    p = SIRS if name == "sirs" else {"beta": 0.4, "gamma": 0.1, "N": 5000,
                                     "I0": 20}
    return [dict(p, beta=0.3 + 0.02 * i) for i in range(n_groups)]


@pytest.mark.parametrize("name,n_groups,n_particles,index", [
    ("sir_cases", 40, 3, [4, 1]), ("sir_cases", 2, 129, None),
    ("seir_age", 3, 5, [96, 2, 50]), ("seir_age", 1, 161, None),
    ("sirs", 5, 33, [3])])
def test_simulate_equals_runs_to_each_time(built, name, n_groups, n_particles,
                                           index):
    gen = d.Generator(name)
    out = []
    for at_once in (True, False):
        sys = d.dust_system_create(gen, _pars(name, n_groups),
                                   n_particles=n_particles,
                                   n_groups=n_groups, dt=0.25, seed=3,
                                   preserve_particle_dimension=True,
                                   preserve_group_dimension=True)
        d.dust_system_set_state_initial(sys)
        if at_once:
            res = d.dust_system_simulate(sys, TIMES, index)
        else:
            res = []
            for t in TIMES:
                d.dust_system_run_to_time(sys, t)
                s = d.dust_system_state(sys)
                res.append(s if index is None else s[np.array(index) - 1])
            res = np.stack(res, axis=-1)
        out.append((res, d.dust_system_state(sys), d.dust_system_time(sys),
                    d.dust_system_rng_state(sys)))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
