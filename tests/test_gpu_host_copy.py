"""Large host operands through the pinned staging: ragged sizes around a piece
(1 MiB) and the smallest staged size, strided and Fortran or C order, columns
longer than a piece, several workspaces on several threads."""
import threading

import numpy as np
import pytest

from csharp_linearalgebra_b200 import Workspace

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(181, 181), (182, 181), (1, 40001), (40001, 1), (131072, 3), (131073, 2), (200003, 2),
                                 (513, 1025), (1023, 1025), (3, 90000)])
@pytest.mark.parametrize("cplx", [False, True])
def test_round_trip(ws, m, n, cplx):
    """A product with a 1 x 1 or identity factor brings every element there and
    back unchanged."""
    rng = np.random.default_rng(m + n)
    a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0)
    one = np.array([[1.0 + (0j if cplx else 0)]])
    if min(m, n) == 1:
        got = ws.multiply(one, a) if m == 1 else ws.multiply(a, one)
    elif n <= 3:
        got = ws.multiply(a, np.eye(n) + (0j if cplx else 0))
    elif m <= 3:
        got = ws.multiply(np.eye(m) + (0j if cplx else 0), a)
    else:
        got = ws.multiply(np.eye(m) + (0j if cplx else 0), a)
    assert np.array_equal(got, a)


def test_factor_leaves_its_input_and_takes_any_layout(ws, orc):
    rng = np.random.default_rng(3)
    big = rng.standard_normal((620, 700))
    for a in (big[:300, :300], np.asfortranarray(big[:400, :300]), big.T[50:350:1, ::2][:, :300]):
        before = a.copy()
        lu = ws.factor_lu(a)
        f, piv, _ = orc.getrf(np.asfortranarray(a), 0)
        assert np.array_equal(lu.factors, f) and np.array_equal(lu.pivots, piv)
        assert np.array_equal(a, before)


def test_workspaces_on_threads():
    failures = []

    def work(seed):
        try:
            rng = np.random.default_rng(seed)
            with Workspace() as w:
                for n in (300, 700, 500):
                    a = rng.integers(-8, 9, (n, n)).astype(float)
                    b = rng.integers(-8, 9, (n, n)).astype(float)
                    if not np.array_equal(w.multiply(a, b), a @ b):
                        failures.append((seed, n))
        except Exception as e:  # reported below
            failures.append(e)

    threads = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
