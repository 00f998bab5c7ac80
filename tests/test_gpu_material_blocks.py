"""The material kernel's block sizes (128 threads, 256 from 100,000 elements,
512 from a million) at the sizes on both sides of the rule, against the same
element body in a batch's blocks: the state and the constraint minima over the
blocks are the same bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("s", [4, 46, 47, 99, 100])
def test_run_matches_batch_blocks(pkg, s, precision):
    with pkg.Lulesh(s, pkg.INIT_V2, precision) as a, pkg.Batch([s], None, pkg.INIT_V2, precision) as b:
        assert a.run(4) == 4
        b.run(4)
        for k in ("x", "xd", "e", "p", "q", "v", "ss"):
            assert np.array_equal(a.get_field(k), b.get_field(0, k)), k
        sa, sb = a.scalars, b.instance(0)[0]
        assert (sa.dtcourant, sa.dthydro, sa.time) == (sb.dtcourant, sb.dthydro, sb.time)
