"""Batches whose launch descriptors, several arrays to one launch, outgrow the
ring they travel through between one array and the next: the first stays where
the launch reads it."""
import numpy as np
import pytest

from csharp_linearalgebra_b200 import Workspace

pytestmark = pytest.mark.gpu

# A product's two tensor maps are 256 bytes, so those of this many matrices in
# one group pass the ring's 4 MiB, behind the products' own descriptors.
COUNT = 17000


def test_products_of_a_batch_beyond_the_ring(orc):
    rng = np.random.default_rng(5)
    mats = []
    for k in range(COUNT):
        n = 2 + k % 2
        a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        mats.append(np.asfortranarray(a * 4.0 ** (k % 5 - 2)))
    with Workspace() as w:
        w.set_workers(1)
        got = w.expm_batched(mats)
        again = w.expm_batched(mats[:300])  # through the ring as it has become
    with Workspace() as w:
        for k in range(0, COUNT, 1000):
            for g, r in zip(got[k:k + 50], w.expm_batched(mats[k:k + 50])):
                assert np.array_equal(g, r)
    for g, r in zip(again, got):
        assert np.array_equal(g, r)
    for k in range(0, COUNT, 500):
        assert np.array_equal(got[k], orc.expm(mats[k])[0])
