"""The cube's set-up on the device against the host's (lulesh_mesh_build), bit
for bit, alone and as instances of a batch: the smallest meshes, sizes on both
sides of a 256-element tile's end, an odd and an ordinary one."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 3, 6, 7, 16, 33, 50)


@pytest.mark.parametrize("init", [1, 2])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_cube_data_match_host_bits(pkg, precision, init):
    scale = np.linspace(0.5, 2.0, len(SIZES))
    with pkg.Batch(list(SIZES), scale, init, precision) as b:
        for i, s in enumerate(SIZES):
            m = pkg.mesh_build(s, init)
            zero = np.zeros(s ** 3)
            e = zero.copy()
            e[0] = m["e0"]
            want = {"x": m["x"], "y": m["y"], "z": m["z"], "volo": m["volo"], "elemMass": m["elem_mass"],
                    "nodalMass": m["nodal_mass"], "v": zero + 1, "p": zero, "q": zero, "ss": zero,
                    "xd": 0 * m["x"], "yd": 0 * m["x"], "zd": 0 * m["x"]}
            with pkg.Lulesh(s, init, precision) as g:
                for k, w in want.items():
                    assert np.array_equal(g.get_field(k), w), (s, k)
                    assert np.array_equal(b.get_field(i, k), w), (s, k)
                assert np.array_equal(g.get_field("e"), e)
                assert np.array_equal(b.get_field(i, "e"), e * scale[i])
                assert g.scalars.deltatime == m["dt0"] and g.scalars.time == 0.0
                if scale[i] == 1.0:
                    assert b.instance(i)[0].deltatime == m["dt0"]
