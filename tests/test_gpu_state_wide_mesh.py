"""The Domain record of a mesh with more elements than nodes (each hexahedron
of a cube listed three times, which the set-up accepts) up and down, between
pinned arrays and pageable ones: every element's value arrives."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NODE, ELEM = ("x", "y", "z", "xd", "yd", "zd"), ("e", "p", "q", "v", "ss")


def tripled_cube(pkg, s):
    m = pkg.mesh_build(s, pkg.INIT_V2)
    ne = s ** 3
    mesh = {k: m[k] for k in "xyz"}
    mesh["nodelist"] = np.tile(m["nodelist"], 3)
    for k in ("lxim", "lxip", "letam", "letap", "lzetam", "lzetap"):
        mesh[k] = np.concatenate([m[k] + i * ne for i in range(3)])
    for k in ("symm_x", "symm_y", "symm_z", "free_surf"):
        mesh[k] = np.zeros(0, np.int32)
    return mesh


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("s", [10, 30])
def test_state_round_trip(pkg, s, precision, pinned):
    torch = pytest.importorskip("torch")
    with pkg.Lulesh.from_mesh(tripled_cube(pkg, s), precision) as g:
        assert g.num_elem > 1024 * -(-g.num_node // 1024)

        def array(k, fill):
            n = g.num_node if k in NODE else g.num_elem
            a = torch.empty(n, dtype=torch.float64, pin_memory=pinned).numpy()
            a[:] = fill(n)
            return a
        rng = np.random.default_rng(s)
        up = {k: array(k, rng.standard_normal) for k in NODE + ELEM}
        g.upload(pkg.Domain(**up, time=0.5, deltatime=2e-6))
        for k in NODE + ELEM:
            assert np.array_equal(g.get_field(k), up[k]), k
        back = pkg.Domain(**{k: array(k, lambda n: np.full(n, -1.0)) for k in NODE + ELEM})
        g.download(back)
        for k in NODE + ELEM:
            assert np.array_equal(getattr(back, k), up[k]), k
