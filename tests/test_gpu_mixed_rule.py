"""The precision form's solves on either side of the rule that chooses between
one launch and blocks with DMMA updates."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


# Forward difference to LAPACK's solve: two backward-stable solutions, each
# within a few n kappa u of the exact one (here kappa < 60).
@pytest.mark.parametrize("n,nrhs,cplx", [(40, 9, False), (40, 30000, False), (200, 300, False), (200, 20000, False),
                                         (50, 20, True), (50, 30000, True), (200, 300, True)])
def test_both_sides(ws, n, nrhs, cplx):
    rng = np.random.default_rng(n + nrhs)
    a = rng.standard_normal((n, n)) / np.sqrt(n) + 3.0 * np.eye(n)
    b = rng.standard_normal((n, nrhs))
    if cplx:
        a = a + 0.5j * rng.standard_normal((n, n)) / np.sqrt(n)
        b = b + 1j * rng.standard_normal((n, nrhs))
    x, info = ws.solve_mixed(a, b)
    want = np.linalg.solve(a, b)
    assert info["backward_error"] <= 8 * U
    err = np.abs(x - want).sum(axis=0).max() / np.abs(want).sum(axis=0).max()
    assert err <= 10 * n * np.linalg.cond(a, 1) * U


def test_many_columns_of_a_large_order(ws):
    """n = 12,000: 512 right-hand sides take 1.3 times the time of 64 (142 ms,
    112), 1.9 times by the one launch, whose CTAs each read the whole factor
    (223, 118)."""
    rng = np.random.default_rng(1)
    n = 12000
    a = rng.standard_normal((n, n)).T / np.sqrt(n)
    a[np.arange(n), np.arange(n)] += 2.0

    least = [np.inf, np.inf]
    panels = [np.asfortranarray(rng.standard_normal((n, nrhs))) for nrhs in (64, 512)]
    for _ in range(4):
        for k, b in enumerate(panels):
            t = time.perf_counter()
            ws.solve_mixed(a, b)
            least[k] = min(least[k], time.perf_counter() - t)
    assert least[1] < 1.6 * least[0]
