"""A batch's panels packed into clusters: matrices of every number of CTAs, in
every mix that fills a cluster or leaves some of it free, as alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# A complex CTA takes up to 256 rows: 1 to 4 CTAs of a cluster of 4 (and of 3).
@pytest.mark.parametrize("orders", [(1000, 1000, 600, 600, 300), (1000, 700, 300, 100, 100, 100), (600, 300, 300, 100),
                                    (300, 300, 300), (90, 40, 70, 2), (1000, 100, 100, 100, 100, 100, 100, 100, 100)])
def test_mixed_heights(ws, orders):
    rng = np.random.default_rng(len(orders))
    mats = []
    for n in orders:
        a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        mats.append(np.asfortranarray(a * (8.0 / np.abs(a).sum(axis=0).max())))
    ws.set_workers(1)
    try:
        got = ws.expm_batched(mats)
    finally:
        ws.set_workers(4)
    for g, a in zip(got, mats):
        assert np.array_equal(g, ws.expm(a))
