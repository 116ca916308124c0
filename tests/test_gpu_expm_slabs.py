"""Single exponentials whose products have too few tiles for the GPU and whose
depth spans several KC slabs: those products run slab-split (two at once in
the Pade evaluation, with beta = 1), bit for bit the oracle's results."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 257, 300, 385, 520])
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("norm", [0.5, 30.0])
def test_expm_matches_oracle(ws, orc, n, cplx, norm):
    from csharp_linearalgebra_b200 import ExpmDiagnostics
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + (1j * rng.standard_normal((n, n)) if cplx else 0)
    a *= norm / np.abs(a).sum(axis=0).max()
    d = ExpmDiagnostics()
    x = ws.expm(a, d)
    ref, info = orc.expm(a)
    assert (d.degree, d.squarings) == (info["degree"], info["squarings"])
    assert np.array_equal(x, ref)
