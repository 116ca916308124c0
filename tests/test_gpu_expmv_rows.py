"""The Taylor kernel over every split of a matrix's rows: batches large enough
that a CTA takes several steps and chunks of rows, against the single calls
(which spread each matrix thinly) and the oracle, bit for bit."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def matrices(rng, orders, cplx):
    out = []
    for n in orders:
        a = rng.standard_normal((n, n)) * (1.5 / math.sqrt(n))
        out.append(np.asfortranarray(a + 1j * rng.standard_normal((n, n)) / math.sqrt(n) if cplx else a))
    return out


@pytest.mark.parametrize("cols", [1, 4, 7, 16, 31])
@pytest.mark.parametrize("cplx", [False, True])
def test_row_splits(ws, orc, cols, cplx):
    rng = np.random.default_rng(100 + cols)
    orders = [1, 2, 15, 16, 17, 31, 33, 47, 64, 65, 96, 97, 112, 113, 127, 129, 160, 193, 224, 225, 257]
    orders = orders * 9 if cols in (4, 7) else orders * 8
    mats = matrices(rng, orders, cplx)
    panels = [np.asfortranarray(rng.standard_normal((n, cols)) + (1j * rng.standard_normal((n, cols)) if cplx else 0))
              for n in orders]
    diags = []
    outs = ws.expmv_batched(mats, panels, 0.75, diags)
    for k in range(21):
        assert np.array_equal(outs[k], ws.expmv(mats[k], panels[k], 0.75))
        ref, info = orc.expmv(mats[k], panels[k], 0.75)
        assert (diags[k].applications, diags[k].early_exits) == (info["applications"], info["early_exits"])
        assert np.array_equal(outs[k], ref)


def test_a_nonfinite_operator_among_row_splits(ws, orc):
    """A nilpotent operator with an infinite entry (finite parameters): the
    explicit skip of zero terms, in every split."""
    rng = np.random.default_rng(7)
    orders = [20, 70, 150, 230] * 40
    mats = matrices(rng, orders, True)
    panels = [np.asfortranarray(rng.standard_normal((n, 8)) + 0j) for n in orders]
    mats[0] = np.zeros((20, 20), complex, order="F")
    mats[0][0, 19] = np.inf
    panels[0][19] = 0.0
    outs = ws.expmv_batched(mats, panels, 0.5)
    for k in range(4):
        ref, _ = orc.expmv(mats[k], panels[k], 0.5)
        assert np.array_equal(outs[k], ref, equal_nan=True)
