"""Fields that the double-float step keeps as pairs of floats, written by the
host: they come back as they went in until a step writes them, and the time
constraints see a strain rate far below the pairs' range as one that moves."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PAIRS = ("vdov", "arealg", "delv_xi", "delv_eta", "delv_zeta", "delx_xi", "delx_eta", "delx_zeta")


def values(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(n) * 10.0 ** rng.uniform(-300, 300, n)
    v[:7] = (0.0, -0.0, 5e-324, 1e308, np.inf, -np.inf, np.nan)
    return v


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("precision", [0, 2])
def test_written_fields_come_back(pkg, precision):
    with pkg.Lulesh(6, pkg.INIT_V2, precision) as g, pkg.Lulesh(6, pkg.INIT_V2, precision) as ref:
        put = {k: values(g.num_elem, i) for i, k in enumerate(PAIRS)}
        for k, v in put.items():
            g.set_field(k, v)
        g.set_field("x", g.get_field("x"))
        for c in (g, ref):
            c.time_increment()
            c.lagrange_nodal()
        for k, v in put.items():
            assert same(g.get_field(k), v), k
        for c in (g, ref):
            c.lagrange_elements()
        for k in PAIRS:
            assert same(g.get_field(k), ref.get_field(k)), k
        g.set_field("vdov", put["vdov"])
        assert same(g.get_field("vdov"), put["vdov"])
        for c in (g, ref):
            assert c.run(2) == 2
        for k in PAIRS:
            assert same(g.get_field(k), ref.get_field(k)), k
        g.set_field("arealg", put["arealg"])
        for c in (g, ref):
            c.lagrange_leapfrog()
        assert same(g.get_field("arealg"), ref.get_field("arealg"))
        g.set_field("arealg", put["arealg"])
        g.run_profiled(1)
        ref.run_profiled(1)
        assert same(g.get_field("arealg"), ref.get_field("arealg"))


@pytest.mark.parametrize("precision", [0, 2])
def test_kept_after_a_step_that_stopped_before_them(pkg, precision):
    """A force launch that finds a bad volume stops the cycle before the
    kinematics: what the host wrote is still there."""
    for call in (lambda g: g.lagrange_leapfrog(), lambda g: g.run(3), lambda g: g.run_profiled(3)):
        with pkg.Lulesh(6, pkg.INIT_V2, precision) as g:
            put = values(g.num_elem, 9)
            g.set_field("vdov", put)
            v = g.get_field("v")
            v[3] = -1.0
            g.set_field("v", v)
            with pytest.raises(pkg.VolumeError):
                call(g)
            assert same(g.get_field("vdov"), put)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("rate", [1e-60, -1e-60, 5e-324, 1e-40])
def test_constraints_of_a_tiny_strain_rate(pkg, rate, precision):
    """dtcourant = arealg / ss and dthydro = dvovmax / (|vdov| + 1e-20) of the
    one element that moves (LULESH-OMP.cc:2820-2915).  Tolerance: a handful of
    pair operations at 2^-46 each, below 1e-12."""
    with pkg.Lulesh(4, pkg.INIT_V2, precision) as g:
        n = g.num_elem
        vdov = np.zeros(n)
        vdov[5] = rate
        g.set_field("vdov", vdov)
        g.set_field("arealg", np.full(n, 3.0))
        g.set_field("ss", np.full(n, 2.0))
        g.calc_time_constraints()
        sc = g.scalars
        assert abs(sc.dtcourant / 1.5 - 1) < 1e-12
        assert abs(sc.dthydro / (g.params.dvovmax / 1e-20) - 1) < 1e-12
