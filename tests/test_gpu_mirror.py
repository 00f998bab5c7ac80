"""The double-float kernels' element arithmetic in packed pairs: against the
oracle on the smallest meshes, on sizes around the warps and blocks of the
launch shapes and on one over a tile's width, and the mirror symmetry that
its sums keep -- a Sedov blast stays bit for bit symmetric about x = y.

Tolerance: a cycle's double-float operations round at 2^-47 (7e-15) of the
quantities they form, a few hundred of them in sequence over these cycles;
1e-11 of each field's largest value is the bar of the other state
comparisons with the oracle (tests/test_gpu_parity.py)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("x", "y", "z", "xd", "yd", "zd", "e", "p", "q", "v", "ss")


@pytest.mark.parametrize("s,cycles", [(1, 8), (2, 20), (3, 20), (11, 12), (32, 6), (65, 4)])
def test_cycles_match_oracle_and_stay_symmetric(pkg, orc, s, cycles):
    o = orc.Oracle(s, orc.INIT_V2)
    rc, _ = o.run(cycles)   # the smallest meshes reach the stop time first
    assert rc == 0
    with pkg.Lulesh(s, pkg.INIT_V2, pkg.FP64) as g:
        assert g.run(cycles) == o.cycle
        got = {k: g.get_field(k) for k in FIELDS}
    for k in FIELDS:
        ref = o.field(k)
        assert np.max(np.abs(got[k] - ref)) <= 1e-11 * max(np.max(np.abs(ref)), 1e-300), k
    n = s + 1
    for a, b in (("x", "y"), ("xd", "yd"), ("z", "z"), ("zd", "zd")):
        assert np.array_equal(got[a].reshape(n, n, n), got[b].reshape(n, n, n).transpose(0, 2, 1)), a
    for k in ("e", "p", "q", "v", "ss"):
        f = got[k].reshape(s, s, s)
        assert np.array_equal(f, f.transpose(0, 2, 1)), k


def test_pair_fields_through_the_accessors(pkg):
    """vdov, arealg and the Q gradients are kept as pairs of floats: a value
    goes in and comes out to the pair's 48 bits, and a value that fits the
    pair comes out as it went in."""
    rng = np.random.default_rng(3)
    with pkg.Lulesh(6, pkg.INIT_V2, pkg.FP64) as g:
        for k in ("vdov", "arealg", "delv_xi", "delx_zeta"):
            v = rng.standard_normal(g.num_elem) * 10.0 ** rng.integers(-6, 6, g.num_elem)
            g.set_field(k, v)
            w = g.get_field(k)
            assert np.max(np.abs(w - v) / np.abs(v)) < 2.0 ** -47, k
            g.set_field(k, w)
            assert np.array_equal(g.get_field(k), w), k
