"""Launch shape of the batched form: the block size and tiles of a batch follow
the CTAs that share an SM, and results agree with the oracle at each shape."""
import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu

CASES = [
    # complex128: three CTAs of 128 threads, 4096-point tiles (direct DFT 2048), every axis
    ([(2048, 2048)], S.Z2Z, 128, 2048),
    ([(256, 4096)], S.Z2Z, 128, 256 + 256),
    ([(4096, 64)], S.Z2Z, 128, 64 + 64),
    ([(61, 128)], S.Z2Z, 128, 2 + 4),
    # complex64: six CTAs of 128 and 4096-point tiles, or three of 256 and 8192 with a long axis
    ([(64, 96)], S.C2C, 128, 2 + 2),
    ([(4096, 64)], S.C2C, 256, 32 + 32),
]


@pytest.mark.parametrize("shapes,prec,threads,tiles", CASES,
                         ids=lambda v: "x".join(map(str, v[0])) if isinstance(v, list) else str(v))
def test_launch_shape(shapes, prec, threads, tiles):
    batch = _sm100.Batch(shapes, prec)
    d = batch.describe()
    assert (d["threads"], d["tiles"]) == (threads, tiles)
    dt = np.complex128 if prec == S.Z2Z else np.complex64
    xs = [o.uniform_input(s, seed=7, dtype=dt) for s in shapes]
    src = [S.DeviceBuffer(x.size, prec) for x in xs]
    dst = [S.DeviceBuffer(x.size, prec) for x in xs]
    for x, b in zip(xs, src):
        b.upload(x)
    batch.execute([b.ptr for b in src], [b.ptr for b in dst])
    batch.status()
    for x, b in zip(xs, dst):
        ref = o.fftn(x.astype(np.complex128), precise=(prec == S.Z2Z))
        assert o.rel_l2(b.download().reshape(x.shape), ref) <= (1e-14 if prec else 1e-6) * np.log2(x.size)
