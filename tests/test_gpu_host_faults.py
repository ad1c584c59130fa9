"""What the transfers do when the host runs short: threads that cannot be started make a smaller
pool, and a set-up that failed leaves nothing half done.  Each case is a process of its own with
tests/host_faults.cpp preloaded; nothing fails on the GPU."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
COMMON = """
import ctypes, sys
import numpy as np
from solar_b200 import _lib, configs
from solar_b200.solver import Solver
faults = ctypes.CDLL(None)
def fault(name, value, kind=ctypes.c_int):
    kind.in_dll(faults, name).value = value
cfg = configs.c2(nx=64, nr=64)
q = np.random.default_rng(0).standard_normal((6, 5, 64, 64, 64)).astype(np.float32).astype(np.float64)
"""


@pytest.fixture(scope="module")
def preload(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("faults") / "host_faults.so")
    subprocess.check_call(["/usr/bin/g++", "-O1", "-fPIC", "-shared", "-o", so, os.path.join(HERE, "host_faults.cpp"), "-ldl"])
    return so


def run(preload, body):
    env = dict(os.environ, LD_PRELOAD=preload, PYTHONPATH=os.path.dirname(HERE), OMP_NUM_THREADS="1", OPENBLAS_NUM_THREADS="1")
    p = subprocess.run([sys.executable, "-c", COMMON + body], env=env, capture_output=True, text=True, timeout=120)
    assert p.returncode == 0, (p.returncode, p.stderr[-2000:])


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("threads", [0, 2])
def test_few_threads_can_be_started(preload, precision, threads):
    run(preload, f"""
with Solver(cfg, precision="{precision}") as s:
    s.norm(4)
    fault("threads_left", {threads})
    s.set_state(q)
    got = s.get_state()
    fault("threads_left", -1)
    np.testing.assert_array_equal(got, q)
""")


def test_float_upload_after_a_failed_first_one(preload):
    """The first upload cannot allocate its pool: an error, and the next upload sets everything up."""
    run(preload, """
with Solver(cfg, precision="fp32") as s:
    s.norm(4)
    fault("fail_new_min", 120, ctypes.c_size_t)     # the pool: a mutex and two condition variables
    fault("fail_new_max", 400, ctypes.c_size_t)
    fault("fail_new", 1)
    try:
        s.set_state(q)
        raise AssertionError("the allocation did not fail")
    except _lib.SolarError as e:
        assert e.status == _lib.SOLAR_ERR_NOMEM, e
    s.set_state(q)
    np.testing.assert_array_equal(s.get_state(), q)
""")


def test_staging_blocks_stay_with_the_process(preload):
    """The pinned blocks (the one mapping with huge pages asked for that appears with the first
    pageable transfer) are left out of a fork."""
    run(preload, """
def advised():
    found, name = set(), None
    for line in open("/proc/self/smaps"):
        first = line.split()[0]
        if "-" in first and not first.endswith(":"):
            name = first
        elif first == "VmFlags:" and "hg" in line.split():
            found.add((name, "dc" in line.split()))
    return found

out = np.empty_like(q)
with Solver(cfg) as s:
    s.norm(4)
    before = {name for name, _ in advised()}
    s.set_state(q)
    s.set_state(q)
    new = {(name, kept) for name, kept in advised() if name not in before}
    assert new and all(kept for _, kept in new), new
""")


def test_staging_that_cannot_be_set_up_is_tried_once(preload):
    run(preload, """
MAP = 9 * 2 << 20                                       # eight blocks of 2 MiB and room to align them
with Solver(cfg) as s:
    s.norm(4)
    fault("fail_mmap", MAP, ctypes.c_size_t)
    for _ in range(3):
        s.set_state(q)
        np.testing.assert_array_equal(s.get_state(), q)
    fault("fail_mmap", 0, ctypes.c_size_t)
    assert ctypes.c_int.in_dll(faults, "failed_mmaps").value == 1
""")
