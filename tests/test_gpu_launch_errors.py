"""A launch that the runtime refuses is reported by its own call and by no
later one."""
import ctypes

import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 64, 32), (60, 50, 18), (97, 8)], ids=["specialised", "generic", "direct"])
def test_refused_launch_leaves_no_error_behind(dims):
    """A capture that was already invalidated (here by a query of the capturing
    stream) refuses the launches of an execute; the plan and the batch built
    afterwards check their own launches and must not meet that error."""
    cu = ctypes.CDLL("libcuda.so.1")
    x = o.uniform_input(dims, seed=5, dtype=np.complex64)
    a, b = S.DeviceBuffer(x.size), S.DeviceBuffer(x.size)
    a.upload(x)
    plan = _sm100.Plan(dims)
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert cu.cuStreamCreate(ctypes.byref(stream), 1) == 0
    assert cu.cuStreamBeginCapture_v2(stream, 1) == 0
    assert cu.cuStreamQuery(stream) != 0
    with pytest.raises(_sm100.Sm100Error):
        plan.execute(a.ptr, b.ptr, 0, 1.0, stream.value)
    assert cu.cuStreamEndCapture(stream, ctypes.byref(graph)) != 0
    assert cu.cuStreamDestroy_v2(stream) == 0
    _sm100.Plan((1009,)).destroy()
    batch = _sm100.Batch([dims])
    batch.execute([a.ptr], [b.ptr])
    batch.status()
    assert o.rel_l2(b.download().reshape(dims), o.fftn(x.astype(np.complex128))) <= 1e-6 * np.log2(x.size)
