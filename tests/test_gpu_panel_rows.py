"""The interchanges of a panel as parallel moves, and U12 behind them: matrices
whose pivots follow prescribed permutations (reversal, cyclic shifts both ways,
every swap with the last row, none), bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def permuted(n, extra, cplx, order):
    """Rows of a matrix that needs no pivoting, in an order that makes partial
    pivoting undo it."""
    rng = np.random.default_rng(n + extra)
    a = rng.uniform(-0.01, 0.01, (n, n + extra)) + (1j * rng.uniform(-0.01, 0.01, (n, n + extra)) if cplx else 0)
    a[np.arange(n), np.arange(n)] += 4.0
    idx = np.arange(n)
    if order == "reversal":
        idx = idx[::-1]
    elif order == "up":
        idx = np.roll(idx, 1)
    elif order == "down":
        idx = np.roll(idx, -1)
    elif order == "blocks":
        idx = np.concatenate([np.roll(b, 5) for b in np.array_split(idx, 3)])
    return a[idx]


@pytest.mark.parametrize("order", ["none", "reversal", "up", "down", "blocks"])
@pytest.mark.parametrize("n,extra,nb", [(2, 0, 16), (17, 3, 16), (40, 0, 32), (65, 7, 64), (100, 0, 32), (200, 33, 64),
                                        (257, 0, 0)])
@pytest.mark.parametrize("cplx", [False, True])
def test_prescribed_interchanges(ws, orc, n, extra, nb, cplx, order):
    a = permuted(n, extra, cplx, order)
    lu = ws.factor_lu(a, nb)
    f, piv, _ = orc.getrf(a, nb)
    assert np.array_equal(lu.pivots, piv)
    assert np.array_equal(lu.factors, f)
    if extra == 0:
        b = np.arange(3.0 * n).reshape(n, 3) + 0j if cplx else np.arange(3.0 * n).reshape(n, 3)
        assert np.array_equal(lu.solve(b), orc.getrs(f, piv, b))
        assert np.array_equal(lu.solve_adjoint(b), orc.getrs(f, piv, b, adjoint=True))
