"""The scale of a real transform is applied to the finished spectrum: the
scaled result is the unscaled one times the factor, rounded once, bit for bit,
for factors that are no power of two and for one below the normal range."""
import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("scale", [1.0 / 3000, 0.7, 3.0e-45])
@pytest.mark.parametrize("dims", [(16,), (30,), (10, 12, 50), (9, 62)], ids=lambda d: "x".join(map(str, d)))
def test_r2c_scale_is_one_rounding(dims, scale, prec):
    rt = np.float64 if prec else np.float32
    x = o.uniform_input(dims, seed=11, dtype=np.complex128 if prec else np.complex64).real.astype(rt)
    x *= rt(1.0e6)
    plan = _sm100.RPlan(dims, prec)
    n = plan.spectrum_elements
    out = []
    for factor in (1.0, scale):
        a, b = S.DeviceBuffer((x.size + 1) // 2, prec), S.DeviceBuffer(n, prec)
        a.upload(np.ascontiguousarray(x).view(np.complex128 if prec else np.complex64))
        plan.r2c(a.ptr, b.ptr, factor)
        out.append(b.download().view(rt))
    assert np.array_equal(out[1], out[0] * rt(scale))
    assert np.any(out[1])
