"""The stage kernel's launch shapes against the FP64 oracle: every tile, radial chunks with
and without a remainder down to one plane, over a radial and a 3-D sound speed (whose c^2
comes through the ring with each plane), in both precisions.

Tolerances are those of the parity suite: FP64 steps 1e-11, FP32 steps 1e-5 per field."""
import numpy as np
import pytest

from solar_b200 import configs
from solar_b200.solver import Solver
from tests.test_gpu_parity import rel_l2

pytestmark = pytest.mark.gpu

NX, NR, NSTEPS = 64, 19, 2
TILES = [(16, 16), (32, 8), (32, 16), (64, 8)]


@pytest.fixture(scope="module")
def cfg():
    return configs.c2(nx=NX, nr=NR)


@pytest.fixture(scope="module")
def state():
    return np.random.default_rng(11).standard_normal((6, 5, NR, NX, NX))


@pytest.fixture(scope="module")
def c2(cfg):
    base = configs.normalise(cfg.model)[1][None, :, None, None]
    return base * np.random.default_rng(12).uniform(0.8, 1.2, (6, NR, NX, NX))


@pytest.fixture(scope="module")
def want(oracle_mod, cfg, state, c2):
    return {on: oracle_mod.Oracle(cfg, c2_3d=c2 if on else None).rk4(state, NSTEPS) for on in (False, True)}


@pytest.mark.parametrize("kchunk", [1, 5, NR])
@pytest.mark.parametrize("tile", TILES)
@pytest.mark.parametrize("precision,nfields,tol", [("fp64", 5, 1e-11), ("fp64", 4, 1e-11), ("fp32", 5, 1e-5), ("fp32", 4, 1e-5)])
@pytest.mark.parametrize("three_d", [False, True])
def test_rk4_at_every_launch_shape(cfg, state, c2, want, three_d, precision, nfields, tol, tile, kchunk):
    with Solver(cfg, precision=precision, nfields=nfields, tile=tile + (kchunk,), c2_3d=c2 if three_d else None) as s:
        s.set_state(state)
        s.rk4(NSTEPS)
        got = s.get_state()
    for m in range(5 - nfields, 5):
        assert rel_l2(got[:, m], want[three_d][:, m]) <= tol, m


def test_rhs_with_3d_sound_speed_and_source(oracle_mod, cfg, state, c2):
    o = oracle_mod.Oracle(cfg, c2_3d=c2)
    o.set_forcing(1, NR // 2)
    with Solver(cfg, c2_3d=c2) as s:
        s.set_forcing(1, NR // 2)
        got, want = s.compute_rhs(state), o.compute_rhs(state)
    for m in range(5):
        assert rel_l2(got[:, m], want[:, m]) <= 1e-12, m
