"""The split force kernel's staged tiles (4 x 32 elements) on cubes whose edge
fills them, leaves one column or row over or falls one short, against the
gathering kernel of a batch, which runs the same element arithmetic: the same
bits."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [64, 65, 66, 95, 96, 97, 127])
def test_staged_matches_gathered(pkg, s):
    with pkg.Lulesh(s, pkg.INIT_V2, pkg.SPLIT) as a, pkg.Batch([s], None, pkg.INIT_V2, pkg.SPLIT) as b:
        assert a.run(3) == 3
        b.run(3)
        for k in ("x", "y", "z", "xd", "yd", "zd", "e", "v"):
            assert np.array_equal(a.get_field(k), b.get_field(0, k)), k
