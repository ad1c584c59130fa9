"""Kernels of the programmatic launch chain start before the kernel in front of them is done: each
calls grid_dependency_wait() before it issues a load, and releases its successor only after it."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "solar_b200", "csrc")


def kernels():
    """(name, body) of every __global__ function, comments left out."""
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\((?:[^()]|\([^()]*(?:\([^()]*\))?[^()]*\))*\)\s*)?(\w+)\s*\(", text):
            start = text.index("{", m.end())
            yield m.group(1), text[start:text.index("\n}\n", start)]


CHAIN = {n: b for n, b in kernels() if "grid_dependency_wait" in b}


def test_the_chain_is_found():
    src = "".join(open(p).read() for p in glob.glob(os.path.join(CSRC, "*.cu*")))
    launched = set(re.findall(r"launch_pdl\(\s*(\w+)", src)) - {"void"}
    assert len(launched) >= 8 and launched <= set(CHAIN), launched - set(CHAIN)


@pytest.mark.parametrize("name", sorted(CHAIN))
def test_waits_before_loads_and_release(name):
    body = CHAIN[name]
    assert body.count("grid_dependency_wait()") == 1
    wait = body.index("grid_dependency_wait()")
    early = [m.group(0) for m in re.finditer(r"(?<!auto )\b(?:issue\w*|one_sided)\(|release_dependents\(", body[:wait])]
    assert not early, early
