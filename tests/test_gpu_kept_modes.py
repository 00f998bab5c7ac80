"""The force kernel's modes kept by the kinematics kernel against modes formed
from the state: writing a field back unchanged makes the kept ones stale, and
the step's results stay the same bits (s = 3, 13 and 20 in one thread per
element and component, s = 33 in one thread per element)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss", "vdov", "arealg")


@pytest.mark.parametrize("precision", [0, 2])
@pytest.mark.parametrize("s,field", [(3, "xd"), (13, "z"), (20, "yd"), (33, "x")])
def test_kept_modes_are_the_states(pkg, s, field, precision):
    with pkg.Lulesh(s, pkg.INIT_V2, precision) as a, pkg.Lulesh(s, pkg.INIT_V2, precision) as b:
        for _ in range(12):
            b.set_field(field, b.get_field(field))
            for g in (a, b):
                g.time_increment()
                g.lagrange_leapfrog()
        for k in FIELDS:
            assert np.array_equal(a.get_field(k), b.get_field(k)), k
        assert a.scalars.time == b.scalars.time
