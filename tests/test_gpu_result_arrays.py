"""Functional steps whose results the caller keeps, in whole or in part, or
drops: each holds its own step's state, and a chain of them ends in the bits
of the main loop."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("s", [6, 30, 60])
def test_kept_results_stay(pkg, s):
    with pkg.Lulesh(s) as g, pkg.Lulesh(s) as ref:
        d, views, copies = g.download(), [], []
        for _ in range(8):
            d = pkg.lulesh(g, d)
            views.append(d.e[::2])
            copies.append(d.e[::2].copy())
        kept = [pkg.lulesh(g, d) for _ in range(3)]
        assert all(np.array_equal(v, c) for v, c in zip(views, copies))
        assert len({id(k.x) for k in kept}) == 3
        ref.run(8)
        want = ref.download()
        for a, b in zip(d.arrays(), want.arrays()):
            assert np.array_equal(a, b)
    assert all(np.array_equal(v, c) for v, c in zip(views, copies))   # the contexts are gone
