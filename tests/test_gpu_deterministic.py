"""Deterministic systems whose stochastic particles are stepped as counts
(engine/discrete.cuh): their kernels run update() alone.  State equal to the
oracle's at every output time, by simulate and by runs to each time, for one
particle, a packed layout and a tile with a remainder."""

import numpy as np
import pytest

import dust2_gb300 as d

pytestmark = pytest.mark.gpu


def pars_of(name, n):
    rs = np.random.default_rng(2)
    if name == "seir_age":
        return [{"R0": r, "contact": rs.gamma(2.0, 1.0, 256) / 16}
                for r in rs.uniform(1.2, 3, n)]
    return [{"N": 1e5, "I0": 20.0, "beta": b, "gamma": 0.1}
            for b in rs.uniform(0.2, 0.5, n)]


@pytest.mark.parametrize("name", ["sir", "sir_cases", "seir_age"])
@pytest.mark.parametrize("n_groups,n_particles", [(1, 1), (70, 1), (2, 131)])
def test_deterministic_matches_oracle(port, name, n_groups, n_particles):
    gen = getattr(d, name)()
    pars = pars_of(name, n_groups)
    times = np.arange(1.0, 8)

    def system():
        s = d.dust_system_create(gen, pars if n_groups > 1 else pars[0],
                                 n_particles=n_particles, n_groups=n_groups,
                                 dt=0.25, seed=1, deterministic=True)
        d.dust_system_set_state_initial(s)
        return s
    s = system()
    words = np.frombuffer(d.dust_system_rng_state(s), dtype="<u8")
    got = np.asarray(d.dust_system_simulate(s, times))
    want, _ = port.discrete_simulate(
        name, np.concatenate([gen.pack_pars(p) for p in pars]), n_groups,
        n_particles, 0.0, 0.25, words, times, deterministic=True)
    n_state = got.shape[0]
    want = want[:times.size * n_groups * n_particles * n_state].reshape(
        times.size, -1, n_state)
    got = got.reshape(n_state, -1, times.size, order="F")
    np.testing.assert_array_equal(got.transpose(2, 1, 0), want)
    s = system()
    for i, t in enumerate(times):
        d.dust_system_run_to_time(s, t)
        state = np.asarray(d.dust_system_state(s))
        np.testing.assert_array_equal(
            state.reshape(n_state, -1, order="F").T, want[i])
