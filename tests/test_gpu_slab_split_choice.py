"""When the products inside an algorithm are split into KC slabs, and when not:
the results are the same bits either way."""
import os
import subprocess
import sys

import numpy as np
import pytest

from csharp_linearalgebra_b200 import _native

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("cplx", [False, True])
def test_the_autotuner_is_asked_inside_algorithms(cplx):
    """A single exponential's products, few tiles of several slabs, are the
    autotuner's to shape when it is on (a class is timed once per process, so
    a fresh one)."""
    code = f"""
import numpy as np
from csharp_linearalgebra_b200 import Workspace
rng = np.random.default_rng(1)
a = rng.standard_normal((600, 600)) + {'1j * rng.standard_normal((600, 600))' if cplx else '0'}
a = np.asfortranarray(a * (20.0 / np.abs(a).sum(axis=0).max()))
with Workspace() as ws:
    plain = ws.expm(a)
    ws.set_autotune(True)
    ws.reset_stats()
    tuned = ws.expm(a)
    trials = ws.stats()["autotune_trials"]
    again = ws.expm(a)
    assert trials >= 1, trials
    assert ws.stats()["autotune_trials"] == trials
    assert np.array_equal(plain, tuned) and np.array_equal(plain, again)
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=ROOT)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("cplx", [False, True])
def test_without_memory_for_the_planes(ws, cplx):
    """Every device allocation of an exponential refused in turn: the planes'
    refusals cost nothing but the split, every other one is reported."""
    rng = np.random.default_rng(2)
    n = 384  # two slabs of 256, and no padding
    a = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
    a = np.asfortranarray(a * (20.0 / np.abs(a).sum(axis=0).max()))
    want = ws.expm(a)
    lib = _native.load()
    reported = unsplit = 0
    for k in range(1, 2000):
        assert lib.tns_inject_allocation_failure(ws.handle, k) == 0
        try:
            got = ws.expm(a)
        except MemoryError:
            reported += 1
            continue
        assert np.array_equal(got, want)
        try:
            ws.multiply(np.eye(2), np.eye(2))  # a refusal that is still to come
        except MemoryError:
            break
        unsplit += 1
    else:
        pytest.fail("no exponential went without a refusal")
    assert reported > 20 and unsplit >= 6
