"""The transposed kernels at the edges of their tiles and radial chunks: both tiles (16 x 16
and 32 x 8), the smallest radius, chunks with remainders and the one-sided rows on a chunk's
boundary, with and without rho, over a radial and a 3-D sound speed.

<L q, mu> = <q, L^T mu> to 1e-11 of |L q| |mu| in double, as in the adjoint suite; in float the
transposed operators agree with the double ones to 1e-5 per field, the FP32 path's target."""
import numpy as np
import pytest

from solar_b200 import configs
from solar_b200.solver import Solver
from tests.test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(16, 16), (32, 17), (48, 19), (48, 41), (64, 23)]


def setup(nx, nr, nfields, three_d):
    cfg = configs.c1(nx=nx, nr=nr)
    rng = np.random.default_rng(nx + nr)
    q, mu = (rng.standard_normal((6, 5, nr, nx, nx)) for _ in range(2))
    if nfields == 4:
        q[:, 0] = mu[:, 0] = 0.0
    c2 = rng.uniform(0.7, 1.3, (6, nr, nx, nx)) if three_d else None
    return cfg, q, mu, c2


@pytest.mark.parametrize("three_d", [False, True])
@pytest.mark.parametrize("nfields", [4, 5])
@pytest.mark.parametrize("nx,nr", SIZES)
def test_dot_products_fp64(nx, nr, nfields, three_d):
    cfg, q, mu, c2 = setup(nx, nr, nfields, three_d)
    with Solver(cfg, nfields=nfields, c2_3d=c2) as s:
        Lq = s.sponge(q, s.bc_rhs(s.compute_rhs(q)))
        Fq = s.filter_exp(q)
        s.set_state(q)
        s.rk4(2)
        Sq = s.get_state()
        for fwd, adj in ((Lq, s.rhs_adjoint(mu)), (Fq, s.filter_adjoint(mu)), (Sq, s.rk4_adjoint(2, mu))):
            a, b = float((fwd * mu).sum()), float((q * adj).sum())
            assert abs(a - b) <= 1e-11 * np.linalg.norm(fwd) * np.linalg.norm(mu), (a, b)


@pytest.mark.parametrize("nx,nr", SIZES)
@pytest.mark.parametrize("nfields", [4, 5])
def test_fp32_matches_fp64(nx, nr, nfields):
    cfg, q, mu, c2 = setup(nx, nr, nfields, True)
    got = {}
    for precision in ("fp64", "fp32"):
        with Solver(cfg, precision=precision, nfields=nfields, c2_3d=c2) as s:
            got[precision] = [s.rhs_adjoint(mu), s.filter_adjoint(mu), s.rk4_adjoint(2, mu)]
    for a, b in zip(got["fp32"], got["fp64"]):
        for m in range(5 - nfields, 5):
            assert rel_l2(a[:, m], b[:, m]) <= 1e-5, m
