"""The real transforms' row-pair kernels at the sizes where they can go wrong:
rows shorter than a lane group, one point over and under a group's step (4
points a lane, 2 to 32 lanes), rows that are their own mirror (even and odd
other axes, axes of length 1 and 2) and row counts around a block.  Same
oracle and tolerances as test_gpu_r2c.py."""
import pytest
from test_gpu_r2c import test_r2c_and_c2r_vs_oracle as check

pytestmark = pytest.mark.gpu

SHAPES = [(4,), (6,), (16,), (18,), (254,), (256,), (258,), (516,), (2, 2), (2, 4, 14), (3, 16), (5, 2, 34),
          (8, 8, 2), (9, 62), (33, 66), (257, 8), (6, 1, 130), (4, 6, 10, 12)]


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_row_pairs(dims, prec):
    check(dims, prec)
