"""Which transfers wake the host threads of an FP64 context: downloads into memory that is not there
yet and uploads once a context has moved 48 MB; the values are the same by every route."""
import mmap
import os

import numpy as np
import pytest

from solar_b200 import configs
from solar_b200.solver import Solver

pytestmark = pytest.mark.gpu


def threads():
    return len(os.listdir("/proc/self/task"))


def fresh(shape):
    """An array whose pages have never been touched."""
    n = int(np.prod(shape)) * 8
    return np.frombuffer(mmap.mmap(-1, n, flags=mmap.MAP_PRIVATE | mmap.MAP_ANONYMOUS), dtype=np.float64).reshape(shape)


@pytest.fixture(scope="module")
def state():
    cfg = configs.c2(nx=48, nr=58)                       # volumes of 1.02 MiB, a state of 32 MB
    with Solver(cfg) as s:                               # whatever the runtime starts by itself
        s.get_state()
    return cfg, np.random.default_rng(7).standard_normal((6, 5, 58, 48, 48))


def test_download_into_touched_memory_is_direct(state):
    cfg, q = state
    out = np.full(q.shape, np.nan)
    with Solver(cfg) as s:
        s.norm(4)
        before = threads()
        s.get_state(out=out)
        assert threads() == before
        s.get_state(out=fresh(q.shape))
        assert threads() > before or len(os.sched_getaffinity(0)) == 1


def test_a_first_small_upload_is_direct(state):
    cfg, q = state
    with Solver(cfg) as s:
        s.norm(4)
        before = threads()
        s.set_state(q)
        assert threads() == before
        s.set_state(q)                                   # 64 MB in all
        assert threads() > before or len(os.sched_getaffinity(0)) == 1


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_partly_touched_results(state, precision):
    cfg, q = state
    q = q.astype(np.float32).astype(np.float64)
    with Solver(cfg, precision=precision) as s:
        for _ in range(3):
            s.set_state(q)
            out = fresh(q.shape)
            out[:2] = np.nan                             # two zones there, four not
            out[3, 2, :20] = np.nan                      # and a part of a volume
            np.testing.assert_array_equal(s.get_state(out=out), q)
            np.testing.assert_array_equal(s.get_state(out=out), q)
            s.set_state(out)
            np.testing.assert_array_equal(s.get_state(), q)
