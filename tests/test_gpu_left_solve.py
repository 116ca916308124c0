"""The transposed and adjoint solves with a chain warp and producers, bit for
bit against the oracle: orders around their 4-, 8- and 16-row phases and their
sixteens, fours and tails, the orders where the rows per phase drop, divisions
outside the reciprocal form's range, and the factored adjoint solve with its
interchanges on both sides of the rule that hands many right-hand sides to
the staged kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 19, 20, 31, 32, 33, 47, 50, 129, 386]


def operands(n, nrhs, cplx, kind="plain"):
    rng = np.random.default_rng(31 * n + nrhs + cplx)

    def part(*shape):
        return rng.uniform(-0.5, 0.5, shape)

    a = part(n, n) / np.sqrt(n) + (1j * part(n, n) / np.sqrt(n) if cplx else 0) + 2.0 * np.eye(n)
    b = part(n, nrhs) + (1j * part(n, nrhs) if cplx else 0)
    if kind == "range":
        b[:, 0] *= 2.0 ** -900
        a[n // 2, n // 2] *= 2.0 ** -1000
        b[n // 3, 1:] = 0.0
    return a, b


def check(ws, orc, n, nrhs, cplx, kind):
    a, b = operands(n, nrhs, cplx, kind)
    kinds = ("lower_unit_transposed",) if cplx else ("upper_transposed", "lower_transposed", "lower_unit_transposed")
    for tri in kinds:
        with np.errstate(all="ignore"):
            assert np.array_equal(ws.solve_triangular(tri, a, b), orc.trsolve(tri, a, b), equal_nan=True), tri


@pytest.mark.parametrize("n", ORDERS)
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["plain", "range"])
def test_orders(ws, orc, n, cplx, kind):
    check(ws, orc, n, 3, cplx, kind)


@pytest.mark.parametrize("n,cplx", [(1500, False), (1700, False), (3000, False), (3300, False), (1490, True), (1600, True)])
def test_large_orders(ws, orc, n, cplx):
    check(ws, orc, n, 2, cplx, "plain")


@pytest.mark.parametrize("n,nrhs,cplx", [(40, 2, False), (40, 2, True), (129, 1200, False), (300, 1000, True),
                                         (300, 3000, False)])
def test_adjoint_solve(ws, orc, n, nrhs, cplx):
    a, b = operands(n, nrhs, cplx)
    a = a[np.random.default_rng(n).permutation(n)]
    lu = ws.factor_lu(a)
    f, piv, _ = orc.getrf(a)
    assert np.array_equal(lu.solve_adjoint(b), orc.getrs(f, piv, b, adjoint=True))
