"""Where a failed simulation of a continuous-time system leaves its time: at
the start of the last of up to 8 parts of the output times, whether the
output was copied at once or in parts."""

import numpy as np
import pytest

import dust2_gb300 as d

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_times,last", [(1, None), (2, 0), (5, 3), (8, 6),
                                          (20, 16)])
def test_time_after_a_failed_simulation(built, n_times, last):
    pars = {"I0": 10, "N": 1000, "beta": 0.4, "gamma": 0.1}
    sys = d.dust_system_create(d.sirode(), pars,
                               ode_control=d.dust_ode_control(max_steps=2))
    d.dust_system_set_state_initial(sys)
    times = 10 * np.arange(1.0, n_times + 1)
    with pytest.raises(d.DustError, match="too many steps"):
        d.dust_system_simulate(sys, times)
    d.dust_system_set_state_initial(sys)
    assert d.dust_system_time(sys) == (0 if last is None else times[last])
