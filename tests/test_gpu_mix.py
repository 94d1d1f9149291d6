"""The generic pass (k_fft_mix) at the sizes where it can go wrong, against
the oracle: every radix alone and as first, middle and last stage, one to
four stages, tiles with a ragged last column, extents that break the 16-byte
alignment of column pairs, single-column tiles, and (batched form) buffers
that start on 8 bytes.

Tolerance: the accuracy bar of the path, relative L2 against the FP64 (long
double for complex128) oracle of 1e-6 * log2 N and 1e-14 * log2 N."""
import math

import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu

# axes last to first: the last is a row pass, the others column passes
SHAPES = [(r, r) for r in range(2, 14)] + [          # one stage, rows and columns, ragged tiles
    (4096,), (2187,), (2401,), (1331,), (2197,), (1000,), (14,), (22, 3),  # single rows, 2 to 4 stages
    (2048, 6), (6, 2048), (1728, 17), (169, 121),   # narrow column tiles; odd extents
    (35, 27, 45), (3, 40, 33), (60, 50, 2), (1, 90, 1), (99, 64, 31 * 2), (384, 7, 18),
    (5, 12, 16), (1200, 1215),                       # long axes in both directions
    (1 << 13,), (1 << 16,), (1 << 18,), (1 << 19,),  # two and three specialised factors
    (13 ** 5,), (1215000,), (3, 5000, 7), (6561, 20),  # two and three generic ones, rows and columns
]


def _tol(n, prec):
    return (1e-6 if prec == S.C2C else 1e-14) * max(1.0, math.log2(max(n, 2)))


@pytest.mark.parametrize("prec", [S.C2C, S.Z2Z])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_generic_pass_matches_oracle(dims, prec):
    dt = np.complex128 if prec == S.Z2Z else np.complex64
    x = o.uniform_input(dims, seed=23, dtype=dt)
    plan = _sm100.Plan(dims, prec)
    a, b = S.DeviceBuffer(x.size, prec), S.DeviceBuffer(x.size, prec)
    for direction in (0, 1):
        a.upload(x)
        plan.execute(a.ptr, b.ptr, direction, 0.25, 0)
        ref = 0.25 * o.fftn(x.astype(np.complex128), sign=1 if direction else -1, precise=(prec == S.Z2Z))
        assert o.rel_l2(b.download().reshape(dims), ref) <= _tol(x.size, prec), direction


@pytest.mark.parametrize("offset", [0, 1])
def test_batch_buffers_on_8_bytes(offset):
    """complex64 transforms whose buffers start `offset` elements past a
    16-byte boundary: the same results as aligned ones, bit for bit."""
    shapes = [(48, 20), (24, 10, 12), (350,), (16, 16), (97, 8)]
    outs = []
    for off in (0, offset):
        b = _sm100.Batch(shapes, S.C2C)
        xs = [o.uniform_input(s, seed=40 + i, dtype=np.complex64) for i, s in enumerate(shapes)]
        src = [S.DeviceBuffer(x.size + 2) for x in xs]
        dst = [S.DeviceBuffer(x.size + 2) for x in xs]
        for x, d in zip(xs, src):
            d.upload(np.concatenate([np.zeros(off, np.complex64), x.ravel()]))
        b.execute([d.ptr + 8 * off for d in src], [d.ptr + 8 * off for d in dst])
        b.status()
        outs.append([d.download()[off:off + x.size] for x, d in zip(xs, dst)])
        for x, y in zip(xs, outs[-1]):
            assert o.rel_l2(y.reshape(x.shape), o.fftn(x.astype(np.complex128))) <= _tol(x.size, S.C2C)
    for y0, y1 in zip(*outs):
        assert np.array_equal(y0, y1)


# both forms of the sums (four output pairs a thread, one), even lengths with
# their middle output, rows and columns, ragged tiles
DIRECT = [(17, 40), (34, 17), (97, 6), (362,), (353, 3), (211, 64, 31), (46, 58, 62), (2, 19), (64, 64, 61)]


@pytest.mark.parametrize("prec", [S.C2C, S.Z2Z])
@pytest.mark.parametrize("dims", DIRECT, ids=lambda d: "x".join(map(str, d)))
def test_direct_pass_matches_oracle(dims, prec):
    test_generic_pass_matches_oracle(dims, prec)
