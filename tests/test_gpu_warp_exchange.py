"""Values that the lanes of a warp hand to one another through shared memory,
each lane's in turn, bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 32), (5, 32), (20, 60), (31, 32), (32, 32), (40, 64)])
@pytest.mark.parametrize("cplx", [False, True])
def test_last_pivot_row_from_every_lane(ws, orc, m, n, cplx):
    """Panels of no more rows than columns, whose last pivot row, of several
    entries, is each row in turn: its lane stores what the others hold."""
    rng = np.random.default_rng(m + n)
    base = rng.uniform(-0.1, 0.1, (m, n)) + (1j * rng.uniform(-0.1, 0.1, (m, n)) if cplx else 0)
    base[np.arange(m), np.arange(m)] += 4.0
    for last in range(m):
        order = np.delete(np.arange(m - 1, -1, -1), 0)  # the other pivots, in reverse
        a = base[np.insert(order, last, m - 1)]
        lu = ws.factor_lu(a, 64)
        f, piv, _ = orc.getrf(a, 64)
        assert np.array_equal(lu.pivots, piv)
        assert np.array_equal(lu.factors, f)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 100])
@pytest.mark.parametrize("cplx", [False, True])
def test_divisors_from_every_lane(ws, orc, n, cplx):
    """Triangles whose diagonal differs in every row: each lane prepares one
    divisor, and every lane divides by all of them in turn."""
    rng = np.random.default_rng(n)

    def part(*shape):
        return rng.uniform(-1.0, 1.0, shape)

    a = part(n, n) / n + (1j * part(n, n) / n if cplx else 0)
    a[np.arange(n), np.arange(n)] = (1.0 + rng.uniform(size=n)) * 3.0 ** rng.integers(-9, 10, n) * \
        (np.exp(2j * np.pi * rng.uniform(size=n)) if cplx else rng.choice([-1.0, 1.0], n))
    for nrhs in (1, 4, 40, 500):  # one column a CTA, and several
        b = part(n, nrhs) + (1j * part(n, nrhs) if cplx else 0)
        for tri in ("upper",) + (() if cplx else ("lower",)):
            assert np.array_equal(ws.solve_triangular(tri, a, b), orc.trsolve(tri, a, b)), (tri, nrhs)


@pytest.mark.parametrize("n", [1, 33, 257, 1500])
@pytest.mark.parametrize("adjoint", [False, True])
def test_long_chains_of_interchanges(ws, orc, n, adjoint):
    """Pivot sequences whose interchanges pass a row along through hundreds of
    others (each with the next row, or all with the last), which the threads
    follow side by side."""
    k = np.arange(n)
    rng = np.random.default_rng(n)
    f = np.eye(n) * 2.0 + rng.uniform(-0.5, 0.5, (n, n)) / n
    b = rng.uniform(-1.0, 1.0, (n, 2))
    for piv in (np.minimum(k + 1, n - 1), np.full(n, n - 1), np.maximum(k, n - 1 - k), rng.integers(k, n)):
        x = np.asfortranarray(b.copy())
        piv = piv.astype(np.int32)
        ff = np.asfortranarray(f)
        ws._call("tns_dgetrs", n, 2, ff.ctypes.data, n, piv.ctypes.data, -1, x.ctypes.data, n, int(adjoint))
        assert np.array_equal(x, orc.getrs(f, piv, b, adjoint=adjoint))
