"""The estimator's one- and two-column products and the one-launch ell chain at
the edges of their layouts (8- and 16-row warps, 16-column tiles, 32-column
groups, the cluster's 1024 columns), bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDERS = [1, 2, 7, 8, 9, 15, 17, 31, 33, 64, 100, 129, 257, 513, 1030]


def matrix(n, cplx, seed):
    rng = np.random.default_rng(seed)
    a = rng.uniform(-1.0, 1.0, (n, n)) + (1j * rng.uniform(-1.0, 1.0, (n, n)) if cplx else 0)
    return a / max(1.0, np.sqrt(n))


@pytest.mark.parametrize("n", ORDERS)
@pytest.mark.parametrize("cplx", [False, True])
def test_products(ws, orc, n, cplx):
    rng = np.random.default_rng(n)
    a = matrix(n, cplx, n)
    for t in (1, 2):
        x = rng.uniform(-1.0, 1.0, (n, t)) + (1j * rng.uniform(-1.0, 1.0, (n, t)) if cplx else 0)
        sparse = np.where(rng.uniform(size=(n, t)) < 0.8, 0.0, x)
        unit = np.zeros((n, t), dtype=x.dtype)
        unit[n // 2, 0] = 1.0
        for panel in (x, sparse, unit):
            for transposed in (False, True):
                assert np.array_equal(ws.multiply_panel(a, panel, transposed), orc.panel(a, panel, transposed))


def test_zero_entries_skip_infinities(ws, orc):
    a = matrix(40, True, 3)
    a[:, 5] = np.inf
    x = np.ones((40, 2), dtype=complex)
    x[5] = 0.0
    assert np.array_equal(ws.multiply_panel(a, x), orc.panel(a, x))


@pytest.mark.parametrize("n", ORDERS)
@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("power,columns", [(1, 1), (3, 2), (8, 2)])
def test_power_estimates(ws, orc, n, cplx, power, columns):
    a = matrix(n, cplx, 10 * n + power)
    r = ws.estimate_power_norm(a, power, columns)
    assert (r.value, r.iterations, r.products) == orc.normest_power(a, power, columns)


@pytest.mark.parametrize("n", [2, 33, 128, 129, 300, 1030])
@pytest.mark.parametrize("norm", [0.012, 0.2, 1.2])
def test_ell_decides_as_the_oracle(ws, orc, n, norm):
    from csharp_linearalgebra_b200 import ExpmDiagnostics
    # Nonnormal: the ell chain, not the norm, decides.
    a = np.triu(np.random.default_rng(n).uniform(0.0, 1.0, (n, n)))
    a *= norm / a.sum(axis=0).max()
    d = ExpmDiagnostics()
    x = ws.expm(a, d)
    ref, info = orc.expm(a)
    assert (d.degree, d.squarings) == (info["degree"], info["squarings"])
    assert np.array_equal(x, ref)
