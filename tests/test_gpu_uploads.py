"""Several uploads in one call: no pinned block is refilled before its last copy is done, also
when that copy belongs to the upload before."""
import numpy as np
import pytest

from solar_b200 import configs
from solar_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("nx,nr", [(32, 20), (64, 48), (64, 129)])
def test_uploads_of_one_call_do_not_mix(nx, nr, precision):
    """SPONGE uploads the right-hand side and the state, CURL three fields, without a wait in
    between.  Both operators are linear and leave zeros where every input is zero, so with one
    input nonzero and of constant value a misplaced volume shows in whole zones."""
    cfg = configs.c1(nx=nx, nr=nr)
    shape = (6, 5, nr, nx, nx)
    zone = np.arange(1.0, 7.0)[:, None, None, None, None]
    field = np.arange(1.0, 6.0)[None, :, None, None, None]
    rhs = np.broadcast_to(8.0 * zone + field, shape).copy()        # one value per volume, exact in float
    axi, aeta, ar = np.random.default_rng(4).standard_normal((3, 6, nr, nx, nx)).astype(np.float32).astype(np.float64)
    with Solver(cfg, precision=precision) as s:
        def alone(m):                                              # the curl of one component
            a = [np.zeros_like(ar)] * 3
            a[m] = (axi, aeta, ar)[m]
            return s.curl(*a)

        parts = [alone(m) for m in range(3)]
        for _ in range(10):
            # v_xi and v_eta are not damped; with a zero state the other fields are not either
            np.testing.assert_array_equal(s.sponge(np.zeros(shape), rhs), rhs)
            np.testing.assert_array_equal(s.sponge(rhs, np.zeros(shape))[:, 1:3], 0.0)
        whole = s.curl(axi, aeta, ar)
        tol = 1e-13 if precision == "fp64" else 1e-5               # sums in another order
        for got, a, b, c in zip(whole, *parts):
            want = a + b + c
            assert np.abs(got - want).max() <= tol * (np.abs(a) + np.abs(b) + np.abs(c)).max()
