"""A batch of thousands of small solves in one group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_many_small_denominators(ws, orc):
    """Thousands of Pade solves in one group, each found by its own item."""
    rng = np.random.default_rng(3)
    mats = [np.asfortranarray(rng.standard_normal((2 + k % 5, 2 + k % 5)) * (1 + 1j)) for k in range(3000)]
    ws.set_workers(1)
    try:
        got = ws.expm_batched(mats)
    finally:
        ws.set_workers(4)
    for k in range(0, 3000, 37):
        assert np.array_equal(got[k], orc.expm(mats[k])[0])
