"""Divisions by a prepared divisor (csrc/divide.cuh), through diagonal solves of
every kernel that uses it, against IEEE division (complex: the oracle's Smith
division): random operands, quotients near the middle between two doubles,
mantissas of all ones, powers of two and their neighbours, the edges of the
range in which the reciprocal is used, and operands outside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def mantissas(rng, size):
    kind = rng.integers(0, 4, size)
    m = 1.0 + rng.integers(0, 2 ** 52, size) * 2.0 ** -52
    m = np.where(kind == 1, 2.0 - rng.integers(1, 4, size) * 2.0 ** -52, m)  # all ones, or nearly
    return np.where(kind == 2, 1.0 + rng.integers(0, 3, size) * 2.0 ** -52, m)  # a power of two, or nearly


def values(rng, size, span):
    """Signed values with exponents to +-span, half of them at its edges."""
    e = rng.integers(-span, span + 1, size)
    edge = rng.choice([-1, 1], size) * (span - rng.integers(0, 3, size))
    e = np.where(rng.uniform(size=size) < 0.5, e, edge)
    return np.ldexp(mantissas(rng, size) * rng.choice([-1.0, 1.0], size), e)


def dividends(rng, d, nrhs, span):
    """Per divisor: random values, and ones whose quotient lies near a midpoint."""
    a = values(rng, (len(d), nrhs), span)
    half = nrhs // 2
    q = np.longdouble(mantissas(rng, (len(d), half))) + np.longdouble(2.0) ** -53
    a[:, :half] = (q * np.longdouble(d)[:, None]).astype(np.float64)
    return a


# Right-hand sides: one launch of one column a CTA and of several, and by blocks.
@pytest.mark.parametrize("n,nrhs", [(1, 900), (7, 60), (32, 2000), (32, 20001), (45, 20001)])
@pytest.mark.parametrize("span", [20, 501, 1020])
def test_real(ws, orc, n, nrhs, span):
    rng = np.random.default_rng(n + nrhs + span)
    d = values(rng, n, span)
    a = dividends(rng, d, nrhs, span)
    a[:, -4:] = [0.0, np.inf, -np.inf, np.nan]
    with np.errstate(all="ignore"):
        want = a / d[:, None]
    # A quotient that is not finite reaches the column's other rows, as a product
    # with the zeros beside the diagonal: there the oracle's answer.
    finite = np.isfinite(want).all(axis=0)
    for tri in ("upper", "lower"):
        got = ws.solve_triangular(tri, np.diag(d), a)
        assert np.array_equal(got[:, finite], want[:, finite]), tri
        assert np.array_equal(got, orc.trsolve(tri, np.diag(d), a), equal_nan=True), tri


@pytest.mark.parametrize("n,nrhs", [(1, 400), (16, 148), (50, 400)])
@pytest.mark.parametrize("span", [20, 501, 1020])
def test_real_transposed(ws, n, nrhs, span):
    """The chain kernel, whose rows' sums are of zeros here (finite operands)."""
    rng = np.random.default_rng(n + nrhs + span)
    d = values(rng, n, min(span, 505))
    a = dividends(rng, d, nrhs, min(span, 505))
    got = ws.solve_triangular("upper_transposed", np.diag(d), a)
    assert np.array_equal(got, a / d[:, None])


@pytest.mark.parametrize("n,nrhs", [(1, 900), (32, 2000), (32, 20001)])
@pytest.mark.parametrize("span", [20, 251, 501])
def test_complex(ws, orc, n, nrhs, span):
    rng = np.random.default_rng(n + nrhs + span)
    d = values(rng, n, span) + 1j * values(rng, n, span)
    a = values(rng, (n, nrhs), span) + 1j * values(rng, (n, nrhs), span)
    a[:, :nrhs // 3] = dividends(rng, d.real, nrhs // 3, span)  # a real dividend
    a[:, -2:] = [0.0, 1j]
    got = ws.solve_triangular("upper", np.diag(d), a)
    assert np.array_equal(got, orc.trsolve("upper", np.diag(d), a), equal_nan=True)
