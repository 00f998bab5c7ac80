"""The material kernel's block sizes (128 threads, 256 from 100,000 elements,
512 from a million) at the sizes on both sides of the rule: its constraint
minima over the blocks are the minima that the separate constraint kernel
takes from the stored fields, from the same values in the same arithmetic, and
the state is the phase calls'."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("s", [4, 46, 47, 99, 100])
def test_leapfrog_matches_phases(pkg, s, precision):
    with pkg.Lulesh(s, pkg.INIT_V2, precision) as a, pkg.Lulesh(s, pkg.INIT_V2, precision) as b:
        rng = np.random.default_rng(s)
        xd = rng.standard_normal(a.num_node)
        for g in (a, b):
            g.set_field("xd", xd)
        for _ in range(2):
            a.time_increment()
            a.lagrange_leapfrog()
            b.time_increment()
            b.lagrange_nodal()
            b.lagrange_elements()
            b.calc_time_constraints()
        for k in ("x", "xd", "e", "p", "q", "v", "ss"):
            assert np.array_equal(a.get_field(k), b.get_field(k)), k
        sa, sb = a.scalars, b.scalars
        assert (sa.dtcourant, sa.dthydro, sa.time) == (sb.dtcourant, sb.dthydro, sb.time)
