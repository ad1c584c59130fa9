"""Per-step norms of changing fields, runs and lengths come from one captured graph: the values are
those of single steps, and a caller that changes them pays for no new graph."""
import time

import numpy as np
import pytest

from solar_b200 import configs
from solar_b200.solver import Solver

pytestmark = pytest.mark.gpu


def test_changing_field_run_and_length():
    cfg = configs.c2(nx=16, nr=24)
    q = np.random.default_rng(6).standard_normal((2, 6, 5, 24, 16, 16))
    with Solver(cfg, nruns=2) as a, Solver(cfg, nruns=2) as b:
        for r in range(2):
            a.set_state(q[r], r)
            b.set_state(q[r], r)
        for field, run, n in ((4, 0, 2), (5, 1, 1), (1, 0, 3), (4, 1, 7), (2, 1, 2)):
            want = []
            for _ in range(n):
                b.rk4(1)
                want.append(b.norm(field, run))
            np.testing.assert_array_equal(a.rk4_norms(n, field=field, run=run), want)


def test_alternating_fields_cost_no_new_graph():
    """Capturing and instantiating a step's graph takes several times as long as a step of this grid
    (0.05 ms); the fastest of 30 calls each, so that a disturbed call does not count."""
    with Solver(configs.c2(nx=16, nr=16)) as s:
        def fastest(fields):
            best = float("inf")
            for k in range(30):
                t = time.perf_counter()
                s.rk4_norms(1, field=fields[k % len(fields)])
                if k >= 4:
                    best = min(best, time.perf_counter() - t)
            return best

        assert fastest([4, 5]) < 1.5 * fastest([4])
