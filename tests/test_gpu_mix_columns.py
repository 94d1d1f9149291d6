"""Column tiles of the generic pass without the bank permutation (at least 8
chunks of 16 bytes a row and 888 tiles) with middle stages: two, three and four
stages, and a ragged last tile, against the oracle.

Tolerance: the accuracy bar of the path, relative L2 against the FP64 (long
double for complex128) oracle of 1e-6 * log2 N and 1e-14 * log2 N."""
import math

import numpy as np
import pytest

import shafft_b200 as S
from oracle import oracle as o
from shafft_b200 import _sm100

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [S.C2C, S.Z2Z])
@pytest.mark.parametrize("dims,stages", [((120, 384, 120), 2), ((384, 126, 117), 3), ((375, 120, 120), 4)])
def test_unpermuted_columns_match_oracle(dims, stages, prec):
    per_chunk = 1 if prec == S.Z2Z else 2
    first = [s for s in _sm100.plan_query(list(dims), prec)["steps"] if s["L"] == dims[0] and not s["in_row"]]
    assert any(len(s["radices"]) == stages and not s["out_row"] and s["W"] // per_chunk >= 8 and s["tiles"] >= 888
               for s in first), first
    n = math.prod(dims)
    x = o.uniform_input(dims, seed=31, dtype=np.complex128 if prec == S.Z2Z else np.complex64)
    plan = _sm100.Plan(dims, prec)
    a, b = S.DeviceBuffer(n, prec), S.DeviceBuffer(n, prec)
    for direction in (0, 1):
        a.upload(x)
        plan.execute(a.ptr, b.ptr, direction, 0.25, 0)
        ref = 0.25 * o.fftn(x.astype(np.complex128), sign=1 if direction else -1, precise=(prec == S.Z2Z))
        tol = (1e-6 if prec == S.C2C else 1e-14) * math.log2(n)
        assert o.rel_l2(b.download().reshape(dims), ref) <= tol, direction
