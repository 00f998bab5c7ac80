"""A batch instance's first time step and energy (lulesh-2.0.3/lulesh-init.cc:
171-182 with the instance's energy factor; LULESH-OMP.cc:3053, :3112), to the
bit, for factors that leave the Sedov values and factors that change them."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 7, 16, 33, 50)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("init", [1, 2])
@pytest.mark.parametrize("factors", [None, [1.0] * 6, [0.5, 1.0, 2.0, 0.7, 1.9, 1.3]])
def test_first_step_and_energy(pkg, factors, init, precision):
    with pkg.Batch(list(SIZES), factors, init, precision) as b:
        for i, s in enumerate(SIZES):
            m = pkg.mesh_build(s, init)
            e0 = m["e0"] * (factors[i] if factors else 1.0)
            cbrt = np.cbrt(m["volo"][0])
            # the C library's cube root is within an ulp of numpy's
            want = 0.5 * cbrt / math.sqrt(2.0 * e0) if init == pkg.INIT_V2 else 1e-7
            sc, origin, status = b.instance(i)
            assert origin == e0 and status == pkg.OK
            assert (sc.time, sc.cycle, sc.dtcourant, sc.dthydro) == (0.0, 0, 1e20, 1e20)
            assert abs(sc.deltatime - want) <= 4 * np.spacing(want)
            if e0 == m["e0"]:
                assert sc.deltatime == m["dt0"]
