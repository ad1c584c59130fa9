"""Host arrays of every kind the transfers tell apart: pageable and pinned, volumes below 1 MiB
(copied as they are), above it (through the pinned blocks) and above one 2 MiB block with a
remainder.  Transfers move values, so FP64 results are equal bit for bit."""
import numpy as np
import pytest
import torch

from solar_b200 import configs
from solar_b200.solver import Solver

pytestmark = pytest.mark.gpu


def pinned(shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy()


@pytest.mark.parametrize("nx,nr", [(32, 20), (64, 33), (64, 129)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_state_in_and_out(nx, nr, precision):
    cfg = configs.c2(nx=nx, nr=nr)
    q = np.random.default_rng(1).standard_normal((6, 5, nr, nx, nx)).astype(np.float32).astype(np.float64)
    with Solver(cfg, precision=precision) as s:
        for src in (q, pinned(q.shape)):
            src[...] = q
            for dst in (np.full(q.shape, np.nan), pinned(q.shape)):
                s.set_state(np.zeros(q.shape))
                s.set_state(src)
                np.testing.assert_array_equal(s.get_state(out=dst), q)


def test_operator_and_gradient_outputs():
    cfg = configs.c2(nx=64, nr=48)
    rng = np.random.default_rng(2)
    q = rng.standard_normal((6, 5, 48, 64, 64))
    with Solver(cfg) as s:
        qp = pinned(q.shape)
        qp[...] = q
        np.testing.assert_array_equal(s.compute_rhs(q), s.compute_rhs(qp))
        s.set_state(q)
        s.set_receivers([[0, 10.5, 20.0, 30.25]])
        a = s.misfit_gradient(2, 2, np.zeros((2, 1)))["grad_c"]        # 9.4 MB, pageable
        b = pinned(a.shape)
        s.set_state(q)
        data = np.zeros((2, 1))
        ptr = lambda x: x.ctypes.data_as(__import__("ctypes").POINTER(__import__("ctypes").c_double))  # noqa: E731
        assert s.lib.solar_gpu_misfit_gradient(s._h, 2, 2, ptr(data), None, ptr(b), None, None) == 0
    assert np.linalg.norm(a) > 0
    assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(a)           # atomics reorder sums


def test_two_uploads_in_one_call():
    """SPONGE uploads two states without a wait in between: the second must not overwrite pinned
    blocks that the first is still being copied out of."""
    cfg = configs.c1(nx=64, nr=48)
    rng = np.random.default_rng(3)
    q, rhs = rng.standard_normal((2, 6, 5, 48, 64, 64))
    qp = pinned(q.shape)
    qp[...] = q
    with Solver(cfg) as s:
        want = s.sponge(qp, rhs)
        for _ in range(5):
            np.testing.assert_array_equal(s.sponge(q, rhs), want)
    # v_xi and v_eta are not damped, the others by sigma(k) q (values of a few units: one rounding)
    np.testing.assert_array_equal(want[:, 1:3], rhs[:, 1:3])
    sigma = np.median((rhs - want)[:, 4] / q[:, 4], axis=(0, 2, 3))
    assert sigma.max() > 0.08
    for m in (0, 3, 4):
        assert np.abs(rhs[:, m] - sigma[None, :, None, None] * q[:, m] - want[:, m]).max() <= 1e-14
