"""Large host operands whose columns are short beside their padding: they cross
without it, from and to arrays with and without gaps between their columns."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1, 40001), (2, 30001), (5, 20011), (57, 700), (65, 3001), (200003, 1)])
@pytest.mark.parametrize("gap", [0, 3])
@pytest.mark.parametrize("cplx", [False, True])
def test_there_and_back(ws, m, n, gap, cplx):
    rng = np.random.default_rng(m + n)
    a = np.full((m + gap, n), np.nan, dtype=np.complex128 if cplx else np.float64, order="F")
    a[:m] = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cplx else 0)
    c = np.full_like(a, 7.0, order="F")
    eye = np.eye(m, dtype=a.dtype, order="F") if m <= 100 else np.ones((1, 1), dtype=a.dtype)
    one, zero = np.array([1.0, 0.0]), np.array([0.0, 0.0])
    scale = [one.ctypes.data, zero.ctypes.data] if cplx else [1.0, 0.0]
    if m <= 100:  # I A
        args = (m, n, m, scale[0], eye.ctypes.data, m, a.ctypes.data, m + gap, scale[1], c.ctypes.data, m + gap)
    else:  # A 1
        args = (m, n, 1, scale[0], a.ctypes.data, m + gap, eye.ctypes.data, 1, scale[1], c.ctypes.data, m + gap)
    ws._call("tns_zgemm" if cplx else "tns_dgemm", *args)
    assert np.array_equal(c[:m], a[:m])
    assert np.all(c[m:] == 7.0)  # what lies between the columns is the caller's


def test_short_columns_do_not_bring_their_padding(ws):
    """A norm of 320 KB as one row of a padded 64 against the same bytes as a
    square: about twice the time (more columns to sum), 24 times with the padding."""
    arrays = [np.ones((200, 200), order="F"), np.ones((1, 40000), order="F")]
    least = [np.inf, np.inf]
    for _ in range(40):
        for k, a in enumerate(arrays):
            t = time.perf_counter()
            ws.one_norm(a)
            least[k] = min(least[k], time.perf_counter() - t)
    assert least[1] < 8 * least[0]
