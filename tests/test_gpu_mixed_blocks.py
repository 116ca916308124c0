"""The precision form around its blocks: orders at the edges of the 64-column
steps and of the 512-column panels, and right-hand-side counts on both sides
of each way to solve (chained, one launch, blocked)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# ||b - A x|| / (||A|| ||x|| + ||b||) by infinity norms: the refinement stops at
# 8 u, and forming the residual here in FP64 adds up to n u of its own.
U = 1.1102230246251565e-16


@pytest.mark.parametrize("n", [5, 63, 64, 65, 127, 129, 191, 513, 577])
@pytest.mark.parametrize("nrhs", [1, 8, 9, 33])
@pytest.mark.parametrize("cplx", [False, True])
def test_orders_and_columns(ws, n, nrhs, cplx):
    rng = np.random.default_rng(n + nrhs)
    a = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
    b = rng.standard_normal((n, nrhs)) + (0j if cplx else 0)
    x, _ = ws.solve_mixed(a, b)
    r = np.abs(a @ x - b).max(axis=0)
    den = np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0)
    assert np.all(r <= (8 + 4 * n) * U * den)


@pytest.mark.parametrize("nrhs", [512, 513])
def test_both_sides_of_the_one_launch_solve(ws, nrhs):
    rng = np.random.default_rng(nrhs)
    a, b = rng.standard_normal((200, 200)), rng.standard_normal((200, nrhs))
    x, _ = ws.solve_mixed(a, b)
    r = np.abs(a @ x - b).max(axis=0)
    den = np.abs(a).sum(axis=1).max() * np.abs(x).max(axis=0) + np.abs(b).max(axis=0)
    assert np.all(r <= (8 + 4 * 200) * U * den)
