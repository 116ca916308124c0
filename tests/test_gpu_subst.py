"""The right-looking solves with the columns in shared memory (1, 2, 4 or 8
per CTA) and the wide batches' blocked form, bit for bit against the oracle at
the edges of their 32-row blocks and column groups, with right-hand sides whose
zeros skip updates and operands outside the reciprocal division's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (2, 5), (31, 2), (32, 3), (33, 1), (64, 9), (65, 600), (95, 17), (127, 300), (257, 4), (1100, 1),
          (300, 2400)]


def operands(n, nrhs, cplx, kind):
    rng = np.random.default_rng(n + 13 * nrhs + 7 * cplx)

    def part(*shape):
        return rng.uniform(-0.5, 0.5, shape)

    a = part(n, n) / np.sqrt(n) + (1j * part(n, n) / np.sqrt(n) if cplx else 0) + 2.0 * np.eye(n)
    b = part(n, nrhs) + (1j * part(n, nrhs) if cplx else 0)
    if kind == "zeros":  # unit vectors and sparse columns
        b[rng.uniform(size=b.shape) < 0.7] = 0.0
        b[:, 0] = 0.0
        b[n // 2, 0] = 1.0
    if kind == "range":
        b[:, ::2] *= 2.0 ** -900
        a[:, n // 3] *= 2.0 ** 520
        a[n // 2, n // 2] *= 2.0 ** -1000
    return a, b


@pytest.mark.parametrize("n,nrhs", SHAPES)
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["plain", "zeros", "range"])
def test_triangles_at_the_edges(ws, orc, n, nrhs, cplx, kind):
    a, b = operands(n, nrhs, cplx, kind)
    for tri in ("upper", "lower_unit") + (() if cplx else ("lower",)):
        with np.errstate(all="ignore"):
            assert np.array_equal(ws.solve_triangular(tri, a, b), orc.trsolve(tri, a, b), equal_nan=True), tri


@pytest.mark.parametrize("n,nrhs", SHAPES)
@pytest.mark.parametrize("cplx", [False, True])
def test_factored_solves(ws, orc, n, nrhs, cplx):
    a, b = operands(n, nrhs, cplx, "plain")
    a = a[np.random.default_rng(n).permutation(n)]  # interchanges to apply
    lu = ws.factor_lu(a)
    f, piv, _ = orc.getrf(a)
    assert np.array_equal(lu.solve(b), orc.getrs(f, piv, b))
    assert np.array_equal(lu.solve_adjoint(b[:, :3]), orc.getrs(f, piv, b[:, :3], adjoint=True))
