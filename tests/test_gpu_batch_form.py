"""Launch shape of the batched form: the block size and tiles of a batch follow
the CTAs that share an SM, and results agree with the oracle at each shape."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

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
def test_launch_shape(shapes, prec, threads, tiles, tmp_path):
    # the default widths: in a process that has none from the tuner
    code = f"import json; from shafft_b200 import _sm100; print(json.dumps(_sm100.Batch({shapes}, {prec}).describe()))"
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, SHAFFT_SM100_TUNE_CACHE=str(tmp_path / "none.txt")))
    assert r.returncode == 0, r.stderr[-2000:]
    d = json.loads(r.stdout)
    assert (d["threads"], d["tiles"]) == (threads, tiles)
    batch = _sm100.Batch(shapes, prec)
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
