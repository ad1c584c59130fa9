"""The transposed filter's load ring gives up under its own switch, says so, and the context goes on;
the switch of one transposed kernel leaves the other's operator alone.  (A wait that runs out with
no load in flight: nothing hangs or faults.)"""
import numpy as np
import pytest

from solar_b200 import _lib, configs
from solar_b200.solver import Solver

pytestmark = pytest.mark.gpu


def inject(s, kernels, polls=1000):
    _lib.check(s.lib.solar_gpu_inject_wait_timeout(s._h, kernels, polls))


@pytest.mark.parametrize("precision,nf", [("fp64", 5), ("fp32", 4)])
@pytest.mark.parametrize("nx", [32, 48])
def test_each_transposed_kernel_has_its_switch_and_name(nx, precision, nf):
    cfg = configs.c1(nx=nx, nr=24)
    q = np.random.default_rng(5).standard_normal((6, 5, 24, nx, nx))
    ops = {"rhs_adjoint": (_lib.SOLAR_KERNEL_ADJ_STAGE, "transposed stage kernel"),
           "filter_adjoint": (_lib.SOLAR_KERNEL_ADJ_FILTER, "transposed filter kernel")}
    tol = 1e-12 if precision == "fp64" else 1e-5          # the transposed exchange adds with atomics
    with Solver(cfg, precision=precision, nfields=nf) as s:
        want = {op: getattr(s, op)(q) for op in ops}

        def same(op):
            assert np.linalg.norm(getattr(s, op)(q) - want[op]) <= tol * np.linalg.norm(want[op])

        for op, (bit, name) in ops.items():
            inject(s, bit)
            with pytest.raises(_lib.SolarError) as e:
                getattr(s, op)(q)
            assert e.value.status == _lib.SOLAR_ERR_TIMEOUT and name in str(e.value)
            for other in ops:
                if other != op:
                    same(other)
            with pytest.raises(_lib.SolarError) as e:
                s.rk4_adjoint(1, q)
            assert e.value.status == _lib.SOLAR_ERR_TIMEOUT
            inject(s, 0, 0)
            for again in ops:
                same(again)
