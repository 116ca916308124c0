"""The right-looking solves on either side of the rule that chooses between one
launch and blocks, bit for bit against the oracle."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def operands(n, nrhs, cplx):
    rng = np.random.default_rng(n + nrhs)

    def part(*shape):
        return rng.uniform(-0.5, 0.5, shape)

    a = part(n, n) / np.sqrt(n) + (1j * part(n, n) / np.sqrt(n) if cplx else 0) + 2.0 * np.eye(n)
    b = part(n, nrhs) + (1j * part(n, nrhs) if cplx else 0)
    return np.asfortranarray(a), np.asfortranarray(b)


# By blocks: few rows and many columns, with the rows of one, two and three
# 128-row blocks; in one launch beside them.
@pytest.mark.parametrize("n,nrhs,cplx", [(5, 20001, False), (33, 20001, False), (130, 36000, False), (300, 30000, False),
                                         (9, 20001, True), (40, 30000, True), (140, 60000, True),
                                         (300, 3000, False), (300, 3000, True), (64, 9000, False)])
def test_both_sides(ws, orc, n, nrhs, cplx):
    a, b = operands(n, nrhs, cplx)
    for tri in ("upper", "lower_unit") + (() if cplx else ("lower",)):
        assert np.array_equal(ws.solve_triangular(tri, a, b), orc.trsolve(tri, a, b)), tri


@pytest.mark.parametrize("n,nrhs,cplx", [(33, 20001, False), (300, 30000, False), (40, 30000, True)])
def test_factored_solve_by_blocks(ws, orc, n, nrhs, cplx):
    a, b = operands(n, nrhs, cplx)
    a = a[np.random.default_rng(n).permutation(n)]
    lu = ws.factor_lu(a)
    f, piv, _ = orc.getrf(a)
    assert np.array_equal(lu.solve(b), orc.getrs(f, piv, b))


def test_large_orders_go_by_blocks(ws):
    """Complex n = 6000: 1776 columns take 1.5 times the time of 592 (48 ms, 32),
    2.3 times (81, 36) while one launch took them, a column or two to a CTA."""
    rng = np.random.default_rng(1)
    n = 6000
    f = np.asfortranarray(rng.standard_normal((n, n)) / 80.0 + 2.0 * np.eye(n) + 0j)

    least = [np.inf, np.inf]
    panels = [np.asfortranarray(rng.standard_normal((n, nrhs)) + 0j) for nrhs in (592, 1776)]
    for _ in range(6):
        for k, b in enumerate(panels):
            x = b.copy(order="F")
            t = time.perf_counter()
            ws._call("tns_zsolve_upper", n, x.shape[1], f.ctypes.data, n, x.ctypes.data, n)
            least[k] = min(least[k], time.perf_counter() - t)
    assert least[1] < 1.9 * least[0]


def test_order_beyond_one_launch(ws, orc):
    """A complex order whose columns do not fit a CTA's shared memory (9664)."""
    n = 9700
    rng = np.random.default_rng(2)
    u, v = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n), rng.uniform(-1, 1, n) / n
    a = np.multiply.outer(v, u).T  # column-major
    a[np.arange(n), np.arange(n)] += 2.0
    b = rng.uniform(-1, 1, (n, 2)) + 1j * rng.uniform(-1, 1, (n, 2))
    for tri in ("upper", "lower_unit"):
        assert np.array_equal(ws.solve_triangular(tri, a, b), orc.trsolve(tri, a, b)), tri
