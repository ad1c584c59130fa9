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


@pytest.mark.parametrize("nx,nr", [(16, 16), (32, 22), (48, 47), (144, 17), (272, 16)])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("fp32", 1e-5)])
def test_default_shapes(oracle_mod, nx, nr, precision, tol):
    """Shapes the library chooses itself: one step, which passes every kernel, where the radial
    chunks of the edge and filter kernels leave remainders (48 x 47), where the filter cuts
    every column in two (32 x 22, the smallest that is cut) and where an edge takes two and
    three segments (144: 72 positions each; 272: 91, 91 and 90)."""
    cfg = configs.c2(nx=nx, nr=nr)
    q = np.random.default_rng(nx).standard_normal((6, 5, nr, nx, nx))
    want = oracle_mod.Oracle(cfg).rk4(q, 1)
    with Solver(cfg, precision=precision, tuned=False) as s:
        s.set_state(q)
        s.rk4(1)
        got = s.get_state()
    for m in range(5):
        assert rel_l2(got[:, m], want[:, m]) <= tol, m


def test_batch_shapes_follow_the_live_runs(oracle_mod):
    """The launch shapes of a batch depend on how many runs are live; every run still equals the oracle's."""
    cfg = configs.c2(nx=32, nr=27)
    steps = [1, 3, 2, 3, 0]
    q = np.random.default_rng(3).standard_normal((len(steps), 6, 5, 27, 32, 32))
    o = oracle_mod.Oracle(cfg)
    with Solver(cfg, nruns=len(steps)) as s:
        for r in range(len(steps)):
            s.set_state(q[r], r)
        s.rk4_runs(steps)
        for r, n in enumerate(steps):
            got, want = s.get_state(r), o.rk4(q[r], n)
            for m in range(5):
                assert rel_l2(got[:, m], want[:, m]) <= 1e-11, (r, m)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_norms_across_runs_fields_and_lengths(precision):
    """The norm is part of the step graph: a change of run or field, a longer ring, an unstored
    field and calls of solar_gpu_norm in between give the norms of single steps, bit for bit."""
    cfg = configs.c2(nx=32, nr=21)
    q = np.random.default_rng(5).standard_normal((2, 6, 5, 21, 32, 32))
    calls = [(0, 4, 2), (0, 4, 3), (1, 4, 2), (1, 5, 6), (0, 1, 1), (0, 2, 4)]
    with Solver(cfg, precision=precision, nfields=4, nruns=2) as s, Solver(cfg, precision=precision, nfields=4, nruns=2) as o:
        for r in range(2):
            s.set_state(q[r], r)
            o.set_state(q[r], r)
        for run, field, n in calls:
            want = []
            for _ in range(n):
                o.rk4(1)
                want.append(o.norm(field, run))
            np.testing.assert_array_equal(s.rk4_norms(n, field, run), want)
            assert s.norm(field, run) == want[-1]
