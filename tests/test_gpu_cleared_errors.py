"""Writing the scalars clears a volume error.  A kinematics launch that stops
at one leaves the geometry kept for the next force launch in parts: blocks
that start after the error was raised keep nothing.  The force launch after
the error is cleared has to form it from the positions: bit for bit what it
gives after the positions are written back unchanged, which drops the kept
geometry.

The mesh is a set of unconnected unit cubes, several times what runs at once, one
of them folded to a negative volume with a positive Jacobian at its centre, so
that the force kernel itself accepts it."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIGNS = np.array([[-1, 1, 1, -1, -1, 1, 1, -1], [-1, -1, 1, 1, -1, -1, 1, 1], [-1, -1, -1, -1, 1, 1, 1, 1]], float)
COUNT, FOLDED = 500_000, 700


def boxes():
    xyz = [np.tile(0.5 * (1 + SIGNS[d]), COUNT) for d in range(3)]
    mesh = dict(zip("xyz", xyz), nodelist=np.arange(8 * COUNT, dtype=np.int32))
    for k in ("lxim", "lxip", "letam", "letap", "lzetam", "lzetap"):
        mesh[k] = np.arange(COUNT, dtype=np.int32)
    for k in ("symm_x", "symm_y", "symm_z", "free_surf"):
        mesh[k] = np.zeros(0, np.int32)
    return mesh, xyz


@pytest.mark.parametrize("precision", [0, 2])
def test_forces_after_cleared_volume_error(pkg, precision):
    mesh, xyz = boxes()
    moved = [1.1 * xyz[0], xyz[1].copy(), xyz[2].copy()]
    fold = slice(8 * FOLDED, 8 * FOLDED + 8)
    moved[1][fold] += SIGNS[0] * SIGNS[1]      # 64 V = 64 (1 - 4/3)
    moved[2][fold] -= SIGNS[0] * SIGNS[2]
    rng = np.random.default_rng(1)
    p = rng.uniform(1.0, 2.0, COUNT)
    out = []
    for rewrite in (False, True):
        with pkg.Lulesh.from_mesh(mesh, precision) as g:
            g.lagrange_elements()              # geometry of the unit cubes kept
            for k, v in zip("xyz", moved):
                g.set_field(k, v)
            g.set_field("p", p)
            with pytest.raises(pkg.VolumeError):
                g.lagrange_elements()
            g.scalars = pkg.Scalars(0.0, 1e-6, 1e20, 1e20, 0)
            if rewrite:
                g.set_field("x", g.get_field("x"))
            g.lagrange_nodal()
            out.append([g.get_field(k) for k in ("xd", "yd", "zd")])
    assert np.max(np.abs(out[0][0])) > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
