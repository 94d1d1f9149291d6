"""Direct-DFT passes on data with an infinite real part: the outputs that are
their own partner in the paired sums (X[0], and X[L/2] of even L) have no sine
part, so their imaginary part is the sum of the finite imaginary parts.  Both
forms of the sums (few rows, many rows), rows and columns, and the batched
form.  Tolerance: the bound of a sum of L terms, L * eps * sum |term|."""
import ctypes

import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu


def _check(x, y, L):
    """x, y: (rows, L), one infinite real part at x[-1, 3]."""
    eps = np.finfo(x.real.dtype).eps
    im = x[-1].imag.astype(np.longdouble)
    bound = L * eps * np.abs(im).sum()
    assert y[-1, 0].real == np.inf
    assert abs(y[-1, 0].imag - im.sum()) <= bound
    if L % 2 == 0:
        assert y[-1, L // 2].real == -np.inf
        assert abs(y[-1, L // 2].imag - (im * (-1.0) ** np.arange(L)).sum()) <= bound
    assert np.isfinite(y[:-1].view(x.real.dtype)).all()


def _input(rows, L, prec):
    x = o.uniform_input((rows, L), seed=L, dtype=np.complex128 if prec else np.complex64)
    x[-1, 3] = complex(np.inf, x[-1, 3].imag)
    return x


@pytest.mark.parametrize("prec", [S.C2C, S.Z2Z])
@pytest.mark.parametrize("columns", [False, True])
@pytest.mark.parametrize("rows,L", [(1, 17), (3, 34), (5000, 17), (3000, 62), (40, 353)])
def test_own_partner_outputs_keep_finite_imaginary_parts(rows, L, columns, prec):
    x = _input(rows, L, prec)
    data = np.ascontiguousarray(x.T) if columns else x
    lib = _sm100.load()
    h = ctypes.c_void_p()
    dims = (ctypes.c_int64 * 2)(*data.shape)
    axes = (ctypes.c_int * 1)(0 if columns else 1)
    assert lib.shafft_sm100_plan_create_axes(ctypes.byref(h), 2, dims, prec, 0, 1, axes) == 0
    a, b = S.DeviceBuffer(x.size, prec), S.DeviceBuffer(x.size, prec)
    a.upload(data)
    assert lib.shafft_sm100_execute(h, ctypes.c_void_p(a.ptr), ctypes.c_void_p(b.ptr), 0, 1.0, None) == 0
    y = b.download().reshape(data.shape)
    lib.shafft_sm100_plan_destroy(h)
    _check(x, np.ascontiguousarray(y.T) if columns else y, L)


@pytest.mark.parametrize("prec", [S.C2C, S.Z2Z])
def test_batched_form(prec):
    shapes = [(17,), (34,), (353,)]
    xs = [_input(1, s[0], prec) for s in shapes]
    src = [S.DeviceBuffer(x.size, prec) for x in xs]
    dst = [S.DeviceBuffer(x.size, prec) for x in xs]
    for x, d in zip(xs, src):
        d.upload(x)
    batch = _sm100.Batch(shapes, prec)
    batch.execute([d.ptr for d in src], [d.ptr for d in dst])
    batch.status()
    for x, d, s in zip(xs, dst, shapes):
        _check(x, d.download().reshape(1, -1), s[0])
