"""shafft_sm100_scale at the edges of its blocks and vectors: odd counts, one
vector over and under a block's 1024, and complex64 data that starts on 8
bytes.  Exact: the factor is a power of two."""
import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,offset", [(0, 0), (0, 1), (1, 0)])
@pytest.mark.parametrize("n", [1, 2, 3, 255, 1023, 1024, 1025, 2047, 2048, 2049, 4097, 100003])
def test_scale_is_exact(n, prec, offset):
    dt = np.complex128 if prec else np.complex64
    x = o.uniform_input((n + offset + 3,), seed=n, dtype=dt)
    d = S.DeviceBuffer(x.size, prec)
    d.upload(x)
    _sm100.scale(d.ptr + offset * x.itemsize, n, prec, 0.125)
    y = x.copy()
    y[offset:offset + n] *= dt(0.125)
    assert np.array_equal(d.download(), y)
