"""Device products with operands read where they lie and with copied ones:
odd and even orders, whole and partial k steps, leading dimensions and bases
on and off 16 bytes, the destination overlapping an operand. Small integers,
so that every sum is exact in any order."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def placed(torch, m, pad, shift):
    """m in a device buffer with `pad` more rows per column, `shift` elements in."""
    rows, cols = m.shape
    ld = rows + pad
    buf = torch.full((shift + ld * cols + 2,), 7.0, dtype=torch.complex128 if np.iscomplexobj(m) else torch.float64,
                     device="cuda")
    view = buf[shift:shift + ld * cols].view(cols, ld)[:, :rows]
    view.copy_(torch.from_numpy(np.ascontiguousarray(m.T)))
    return buf, view, buf.data_ptr() + shift * buf.element_size(), ld


@pytest.mark.parametrize("m,n,k", [(2, 2, 16), (64, 96, 32), (130, 66, 48), (129, 66, 48), (130, 65, 48), (130, 66, 47),
                                   (512, 512, 512), (1, 1, 1)])
@pytest.mark.parametrize("pad,shift", [(0, 0), (2, 0), (1, 0), (0, 1), (2, 2)])
@pytest.mark.parametrize("cplx", [False, True])
def test_products(ws, m, n, k, pad, shift, cplx):
    import torch
    rng = np.random.default_rng(m * n + k)

    def draw(r, c):
        x = rng.integers(-8, 9, (r, c)).astype(float)
        return x + 1j * rng.integers(-8, 9, (r, c)) if cplx else x
    a, b, c = draw(m, k), draw(k, n), draw(m, n)
    abuf, av, pa, lda = placed(torch, a, pad, shift)
    bbuf, bv, pb, ldb = placed(torch, b, pad, shift)
    cbuf, cv, pc, ldc = placed(torch, c, pad, shift)
    before = abuf.clone(), bbuf.clone()
    torch.cuda.synchronize()
    from csharp_linearalgebra_b200 import _native
    lib = _native.load()
    if cplx:
        al, be = (np.array([x, 0.0]) for x in (2.0, -1.0))
        rc = lib.tns_zgemm_device(ws._h, m, n, k, al.ctypes.data_as(C.c_void_p), pa, lda, pb, ldb,
                                  be.ctypes.data_as(C.c_void_p), pc, ldc)
    else:
        rc = lib.tns_dgemm_device(ws._h, m, n, k, 2.0, pa, lda, pb, ldb, -1.0, pc, ldc)
    assert rc == 0
    assert np.array_equal(cv.cpu().numpy().T, 2.0 * (a @ b) - c)
    assert torch.equal(abuf, before[0]) and torch.equal(bbuf, before[1])


def test_destination_is_an_operand(ws):
    import torch
    from csharp_linearalgebra_b200 import _native
    a = np.random.default_rng(5).integers(-8, 9, (256, 256)).astype(float)
    buf, view, p, ld = placed(torch, a, 0, 0)
    torch.cuda.synchronize()
    assert _native.load().tns_dgemm_device(ws._h, 256, 256, 256, 1.0, p, ld, p, ld, 0.0, p, ld) == 0
    assert np.array_equal(view.cpu().numpy().T, a @ a)
