"""Launch shapes of a batch by hand: the shape that a batch starts with can be
set again, and asking for more blocks than it takes gives it."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("sizes", [[64, 60, 70, 66], [20, 17]])
def test_default_shapes_can_be_set(pkg, sizes, precision):
    cls = 2 if precision == pkg.SPLIT and max(sizes) >= 48 else 0   # FP64 ensembles are one class
    with pkg.Batch(sizes, None, pkg.INIT_V2, precision) as b:
        for kernel in pkg.BATCH_KERNELS:
            name = f"class{cls}/{kernel}"
            start = b.tuning()[name]
            b.set_tuning(cls, kernel, block=64, blocks_per_sm=1)
            assert b.tuning()[name] != start
            b.set_tuning(cls, kernel, block=start["block"], blocks_per_sm=1_000_000)
            assert b.tuning()[name] == start, name
