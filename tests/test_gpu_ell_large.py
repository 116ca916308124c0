"""The ell test's chain ||abs(A)^p||_1 at orders whose row vector does not fit one
launch (above 5376): the degree and squarings of an exponential that they alone
decide. A has A^2 = 0 in 2 x 2 blocks [[c, -c], [c, -c]], so every norm of its
powers is zero or that of its largest block and only abs(A)'s powers call for
scaling: what the block alone decides."""
import numpy as np
import pytest

from csharp_linearalgebra_b200 import ExpmDiagnostics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5376, 5377, 6001])  # one launch, and one per pass
def test_degree_and_squarings(ws, orc, n):
    rng = np.random.default_rng(n)
    a = np.zeros((n, n), order="F")
    pairs = rng.permutation(n)[:200].reshape(-1, 2)
    pairs[0] = sorted((3, n - 1))
    used = {3, n - 1}
    largest = 40.0
    for k, (i, j) in enumerate(pairs):
        if k and (i in used or j in used):
            continue
        c = largest if k == 0 else rng.uniform(0.01, 30.0)
        a[i, i], a[i, j], a[j, i], a[j, j] = c, -c, c, -c
    diag = ExpmDiagnostics()
    ws.expm(a, diag)
    info = orc.expm(np.array([[largest, -largest], [largest, -largest]]))[1]
    assert (diag.degree, diag.squarings) == (info["degree"], info["squarings"])
    assert diag.squarings > 0
