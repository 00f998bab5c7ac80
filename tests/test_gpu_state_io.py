"""The Domain record up and down on both sides of the staging limit (pageable
arrays through the pinned buffer in one kernel up to s = 25, larger ones field
by field), and between a kernel and pinned arrays:
every bit comes back, arrays left out stay as they are, read-only and strided
inputs are taken, and the scalars that a call does not set keep their values."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NODE, ELEM = ("x", "y", "z", "xd", "yd", "zd"), ("e", "p", "q", "v", "ss")


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("s", [1, 2, 5, 17, 18, 25, 26])
def test_state_round_trip(pkg, s, precision):
    rng = np.random.default_rng(s)
    with pkg.Lulesh(s, pkg.INIT_V2, precision) as g:
        nn, ne = g.num_node, g.num_elem
        g.scalars = pkg.Scalars(0.25, 1e-6, 3.0, 4.0, 7)
        a = {k: rng.standard_normal(nn if k in NODE else ne) for k in NODE + ELEM}
        a["x"].setflags(write=False)
        a["yd"] = np.repeat(a["yd"], 2)[::2]
        g.upload(pkg.Domain(**a, time=0.5, deltatime=2e-6))
        sc = g.scalars
        assert (sc.time, sc.deltatime, sc.dtcourant, sc.dthydro, sc.cycle) == (0.5, 2e-6, 3.0, 4.0, 7)
        d = g.download()
        for k in NODE + ELEM:
            assert np.array_equal(getattr(d, k), a[k]), k
            assert np.array_equal(g.get_field(k), a[k]), k
        assert (d.time, d.deltatime) == (0.5, 2e-6)

        # some fields only, through the C call
        lib, z, q = pkg.load_library(), rng.standard_normal(nn), rng.standard_normal(ne)
        def p(v):
            return v.ctypes.data_as(C.POINTER(C.c_double))
        args = [None] * 11
        args[2], args[8] = p(z), p(q)
        assert lib.lulesh_upload_domain(g._h, *args, 0.75, 3e-6) == 0
        a["z"], a["q"] = z, q
        back = {k: np.full(nn if k in NODE else ne, -1.0) for k in NODE + ELEM}
        out = [None if k == "zd" else p(back[k]) for k in NODE + ELEM]
        t = C.c_double()
        assert lib.lulesh_download_domain(g._h, *out, C.byref(t), None) == 0
        assert t.value == 0.75 and np.all(back["zd"] == -1.0)
        for k in NODE + ELEM:
            if k != "zd":
                assert np.array_equal(back[k], a[k]), k


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("s,skip", [(9, 0), (18, 0), (18, 1), (31, 1)])
def test_pinned_arrays(pkg, s, skip, precision):
    """Pinned arrays, read and written by the kernel itself: aligned to a value
    only (skip), one field left out, one pageable among them."""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(s)
    with pkg.Lulesh(s, pkg.INIT_V2, precision) as g:
        def pinned(k):
            n = g.num_node if k in NODE else g.num_elem
            t = torch.empty(n + skip, dtype=torch.float64, pin_memory=True)
            return t, t.numpy()[skip:]
        keep = {k: pinned(k) for k in NODE + ELEM}
        a = {k: v for k, (_, v) in keep.items()}
        for v in a.values():
            v[:] = rng.standard_normal(v.size)
        g.upload(pkg.Domain(**a, time=0.5, deltatime=2e-6))
        for k in NODE + ELEM:
            assert np.array_equal(g.get_field(k), a[k]), k
        back = {k: pinned(k) for k in NODE + ELEM}
        out = pkg.Domain(**{k: v for k, (_, v) in back.items()})
        out.p = None
        back["p"][1][:] = -1.0
        g.download(out)
        for k in NODE + ELEM:
            assert np.array_equal(back[k][1], a[k] if k != "p" else np.full(g.num_elem, -1.0)), k
        assert (out.time, out.deltatime) == (0.5, 2e-6)
        mixed = pkg.Domain(**{k: v.copy() if k == "q" else v for k, (_, v) in back.items()})
        mixed.q[:] = 7.0
        g.upload(mixed)
        for k in NODE + ELEM:
            assert np.array_equal(g.get_field(k), getattr(mixed, k)), k
