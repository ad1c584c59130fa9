"""The source's clock over the phases of a split step: it advances with the filter that ends the
step (timestep.f90:82), not before, and FILTER_EXP alone leaves it."""
import numpy as np
import pytest

from solar_b200 import _lib, configs
from solar_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("tail", [[5], [6, 7]])
@pytest.mark.parametrize("parts", [False, True])
def test_clock_between_the_phases_of_a_step(precision, tail, parts):
    cfg = configs.c2(nx=32, nr=24)
    with Solver(cfg, precision=precision) as s:
        s.set_forcing(_lib.SOLAR_FORCING_ANALYTIC, 12)
        s.set_clock(0.25, 3)
        for step in range(2):
            before = s.get_clock()
            for phase in range(5):
                if parts:
                    for part in range(2):
                        _lib.check(s.lib.solar_gpu_step_phase_part(s._h, phase, part))
                        assert s.get_clock() == before
                else:
                    _lib.check(s.lib.solar_gpu_step_phase(s._h, phase))
                assert s.get_clock() == before
            for phase in tail:
                assert s.get_clock() == before
                _lib.check(s.lib.solar_gpu_step_phase(s._h, phase))
            assert s.get_clock() == (before[0] + cfg.dt, before[1] + 1)


def test_clock_set_between_phases_is_the_one_that_advances():
    cfg = configs.c2(nx=32, nr=24)
    with Solver(cfg) as s:
        s.set_forcing(_lib.SOLAR_FORCING_ANALYTIC, 12)
        s.set_clock(0.25, 3)
        for phase in range(5):
            _lib.check(s.lib.solar_gpu_step_phase(s._h, phase))
        s.set_clock(0.75, 9)
        _lib.check(s.lib.solar_gpu_step_phase(s._h, 5))
        assert s.get_clock() == (0.75 + cfg.dt, 10)


def test_operators_leave_the_clock():
    cfg = configs.c2(nx=32, nr=24)
    q = np.zeros((6, 5, 24, 32, 32))
    with Solver(cfg) as s:
        s.set_forcing(_lib.SOLAR_FORCING_ANALYTIC, 12)
        s.set_clock(0.25, 3)
        s.filter_exp(q)
        s.compute_rhs(q)
        assert s.get_clock() == (0.25, 3)
        s.rk4(4)
        assert s.get_clock()[1] == 7
