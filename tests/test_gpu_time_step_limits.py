"""TimeIncrement (LULESH-OMP.cc:557-604) next to the largest doubles: four
times the step overflows, and two thirds of it is still what remains to be
taken."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("dt", [5e307, 4.4e307, 4e307, 1.0, 3e-7])
def test_two_thirds_of_the_last_step(pkg, dt, precision):
    p = pkg.default_parameters()
    p.stoptime = 1e308 if dt > 1e300 else 1.2 * dt
    target, want = p.stoptime, dt
    if dt < target < 4.0 * dt / 3.0:
        target = 2.0 * dt / 3.0
    want = min(target, dt)
    with pkg.Lulesh(3, pkg.INIT_V2, precision, p) as g:
        g.scalars = pkg.Scalars(0.0, dt, 1e20, 1e20, 0)
        g.time_increment()
        assert g.scalars.deltatime == want
