"""Performance cases of the Lagrange leapfrog step, through the package's public calls.

Each case is one kind of program that uses the library:

* ``run``    the main loop: the state of a checkpoint goes up, ``run`` advances
             it some cycles (or to the stop time), the state comes back;
* ``step``   the functional step over host arrays, one cycle per call, as a
             host program that owns the Domain record drives it;
* ``phases`` one cycle through the separate phase calls;
* ``batch``  a seeded ensemble of independent problems, created, run and read.

Two initial states: ``origin`` is the Sedov problem at t = 0 (all energy in
one element, scaled by a seeded factor as the ensembles draw it), ``flow`` a
state in mid-blast: a radial velocity, displacement and energy profile with
seeded ripples inside a shock radius, and cold gas at rest outside it.
"""
import importlib
import math

import numpy as np
import torch

LULESH1, LULESH2 = 1, 2                       # initial conditions
ORDER = {"fp64": 0, "split": 1, "ieee": 2}    # precision modes of the library
NODE, ELEM = ("x", "y", "z", "xd", "yd", "zd"), ("e", "p", "q", "v", "ss")
EXTENT = 1.125                                # edge of the Sedov cube


def package():
    return importlib.import_module("lulesh-accelerate_gb300")


def listed():
    return [
        # one cycle over host arrays of a tiny mesh: calls, copies and launches, hardly any arithmetic
        dict(name="step_s8", kind="step", s=8, prec="fp64", state="flow"),
        # the published LULESH 1.0 table's small problem, start to finish: 593 short cycles
        dict(name="run_s10_full", kind="run", s=10, prec="fp64", state="origin", init=LULESH1, cycles=0),
        # the parity configuration, LULESH 2.0 at s=30 to its stop time: 932 cycles
        dict(name="run_s30_full", kind="run", s=30, prec="fp64", state="origin", init=LULESH2, cycles=0),
        # one cycle through the phase calls, in split precision, on an odd size
        dict(name="phases_s47_split", kind="phases", s=47, prec="split", state="flow"),
        # a mesh given by its lists (renumbered, so nothing is structured)
        dict(name="run_s37_unstructured", kind="run", s=37, prec="fp64", state="flow", cycles=100, mesh="lists"),
        # LULESH 2.0's default material regions with their repeated equation of state
        dict(name="run_s64_regions", kind="run", s=64, prec="fp64", state="flow", cycles=60, regions=11),
        # an ordinary run in every-operation-IEEE arithmetic
        dict(name="run_s45_ieee", kind="run", s=45, prec="ieee", state="flow", cycles=60),
        # an ordinary size in mid-blast
        dict(name="run_s90", kind="run", s=90, prec="fp64", state="flow", cycles=60),
        # an ensemble of small uneven problems, each to its own stop time
        dict(name="batch_small_split", kind="batch", prec="split", cycles=0,
             sizes="9,24,13,17,21,8,30,26,11,19,28,15,22,12,27,10"),
        # an ensemble of uneven problems in FP64, a stretch of their cycles
        dict(name="batch_fp64", kind="batch", prec="fp64", cycles=300, sizes="16,41,27,56,33,48,22,37"),
        # the benchmark's mesh, the largest single problem, in both precisions
        dict(name="run_s192", kind="run", s=192, prec="fp64", state="flow", cycles=30),
        dict(name="run_s192_split", kind="run", s=192, prec="split", state="flow", cycles=50),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "step", "phases", "batch"])
    prec = rng.choice(["fp64", "fp64", "split", "split", "ieee"])
    if kind == "batch":
        sizes = [log_int(rng, 8, 56) for _ in range(rng.randint(3, 14))]
        return dict(kind="batch", prec=prec, sizes=",".join(map(str, sizes)), cycles=rng.randint(60, 300))
    if kind == "step":
        return dict(kind="step", s=log_int(rng, 6, 100), prec=prec, state="flow")
    if kind == "phases":
        return dict(kind="phases", s=log_int(rng, 6, 150), prec=prec, state="flow")
    s = log_int(rng, 6, 180)
    case = dict(kind="run", s=s, prec=prec, state="flow",
                cycles=rng.randint(20, max(20, min(200, 100_000_000 // s ** 3 // 2))))
    extra = rng.choice(["", "", "lists", "regions", "origin"])
    if extra == "lists" and s <= 60:
        case["mesh"] = "lists"
    elif extra == "regions":
        case["regions"] = rng.randint(2, 21)
    elif extra == "origin":
        case.update(state="origin", init=rng.choice([LULESH1, LULESH2]))
    return case


# ---- inputs ---------------------------------------------------------------

def device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def cube(s, dev):
    """The Sedov cube: coordinates [3, nodes] and the corner nodes [8, elements]."""
    n = s + 1
    t = EXTENT * torch.arange(n, dtype=torch.float64, device=dev) / s
    z, y, x = torch.meshgrid(t, t, t, indexing="ij")
    i = torch.arange(s, device=dev)
    p, r, c = torch.meshgrid(i, i, i, indexing="ij")
    base = ((p * n + r) * n + c).reshape(-1)
    nodes = torch.stack([base + d for d in (0, 1, n + 1, n, n * n, n * n + 1, n * n + n + 1, n * n + n)])
    return torch.stack([x.reshape(-1), y.reshape(-1), z.reshape(-1)]), nodes


def renumbering(s, seed):
    rng = np.random.default_rng([seed, 7])
    return rng.permutation((s + 1) ** 3), rng.permutation(s ** 3)


def hex_volume(c):
    """Volumes of hexahedra with corners c [3, 8, elements]."""
    def triple(a, b, d):
        return (a * torch.linalg.cross(b, d, dim=0)).sum(0)

    def e(i, j):
        return c[:, i] - c[:, j]
    return (triple(e(3, 1) + e(7, 2), e(6, 3), e(2, 0)) + triple(e(4, 3) + e(5, 7), e(6, 4), e(7, 0)) +
            triple(e(1, 4) + e(2, 5), e(6, 1), e(5, 0))) / 12


class State:
    """The Domain record of a case's initial state, as 64-bit tensors, with its clock."""

    def __init__(self, case, seed):
        dev, s = device(), case["s"]
        rng = np.random.default_rng([seed, s])
        factor = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
        pos, self.nodes = cube(s, dev)
        self.s, self.vol0 = s, hex_volume(pos[:, self.nodes])
        zero = torch.zeros(s ** 3, dtype=torch.float64, device=dev)
        vel = torch.zeros_like(pos)
        self.e, self.p, self.q, self.v, self.ss = zero.clone(), zero.clone(), zero.clone(), zero + 1, zero.clone()
        self.symm = (pos == 0)
        self.cycle = 0
        if case["state"] == "origin":
            first = 3.948746e7 * (factor if case["init"] == LULESH1 else factor * (s / 45.0) ** 3)
            self.e[0] = first
            self.dt = 1e-7 if case["init"] == LULESH1 else 0.5 * float(self.vol0[0]) ** (1 / 3) / math.sqrt(2 * first)
        else:
            radius, width = rng.uniform(0.35, 0.6), 0.05
            wave = torch.tensor(rng.uniform(2.0, 9.0, (4, 3)), device=dev)
            phase = rng.uniform(0.0, 2 * math.pi, 4)

            def profile(r):   # 1 inside the shock, falling to exactly 0 ahead of it
                return (torch.clamp((radius + width - r) / (2 * width), 0, 1) ** 2) * (r < radius + width)

            def ripple(x):
                return sum(torch.sin((wave[i, :, None] * x).sum(0) + phase[i]) for i in range(4)) / 4

            r = pos.norm(dim=0)
            a, w = profile(r), ripple(pos)
            speed = 100.0 * math.sqrt(factor)
            vel = pos / radius * a * speed * (1 + 0.1 * w)
            pos = pos * (1 + 0.04 * a * (1 + 0.2 * w))
            corners = pos[:, self.nodes]
            self.v = hex_volume(corners) / self.vol0
            mid = corners.mean(1)
            b = profile(mid.norm(dim=0))
            self.e = 8e3 * factor * b * (1.2 - mid.norm(dim=0) / radius).clamp(min=0.2) * (1 + 0.1 * ripple(mid))
            self.p = (2.0 / 3.0) * self.e / self.v
            self.q = 50.0 * factor * b * (1 - b)
            self.ss = torch.sqrt((10.0 / 9.0) * self.e / self.v).clamp(min=.333333e-18)
            self.dt = 0.05 * EXTENT / s / (3 * speed)
        if case.get("mesh") == "lists":
            pn, pe = (torch.from_numpy(k).to(dev) for k in renumbering(s, seed))
            at = torch.empty_like(pn)
            at[pn] = torch.arange(len(pn), device=dev)
            pos, vel, self.symm = pos[:, pn], vel[:, pn], self.symm[:, pn]
            self.nodes, self.vol0 = at[self.nodes[:, pe]], self.vol0[pe]
            for k in ELEM:
                setattr(self, k, getattr(self, k)[pe])
        self.x, self.y, self.z = pos
        self.xd, self.yd, self.zd = vel


def neighbours(s, case, seed):
    """Face neighbours [6, elements] (xi-, xi+, eta-, eta+, zeta-, zeta+), an element itself where it has none."""
    k = np.arange(s ** 3)
    at = np.stack([k % s, (k // s) % s, k // (s * s)])
    out = np.empty((6, s ** 3), dtype=np.int64)
    for d, step in enumerate((1, s, s * s)):
        out[2 * d] = np.where(at[d] > 0, k - step, k)
        out[2 * d + 1] = np.where(at[d] < s - 1, k + step, k)
    if case.get("mesh") == "lists":
        _, pe = renumbering(s, seed)
        inv = np.empty_like(pe)
        inv[pe] = k
        out = inv[out[:, pe]]
    return out


def create(case, seed, st):
    lib, prec = package(), ORDER[case["prec"]]
    if case.get("mesh") != "lists":
        return lib.Lulesh(case["s"], case.get("init", LULESH2), prec)
    s = case["s"]
    pos, _ = cube(s, torch.device("cpu"))
    pos = pos[:, torch.from_numpy(renumbering(s, seed)[0])].numpy()
    mesh = dict(zip("xyz", pos), nodelist=st.nodes.t().reshape(-1).cpu().numpy())
    mesh.update(zip(("lxim", "lxip", "letam", "letap", "lzetam", "lzetap"), neighbours(s, case, seed)))
    for d, k in enumerate(("symm_x", "symm_y", "symm_z")):
        mesh[k] = np.flatnonzero(pos[d] == 0)
    mesh["free_surf"] = np.flatnonzero((pos == EXTENT).any(0))
    return lib.Lulesh.from_mesh(mesh, prec)


def pinned(t):
    a = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    return a.copy_(t).numpy()


def prepare(case, seed):
    lib = package()
    if case["kind"] == "batch":
        sizes = [int(k) for k in case["sizes"].split(",")]
        factors = np.exp(np.random.default_rng([seed, 3]).uniform(math.log(0.5), math.log(2.0), len(sizes)))
        return dict(case=case, sizes=sizes, factors=factors)
    st = State(case, seed)
    ctx = create(case, seed, st)
    if case.get("regions"):
        ctx.set_regions(case["regions"])
    start = lib.Domain(**{k: pinned(getattr(st, k)) for k in NODE + ELEM}, time=0.0, deltatime=st.dt)
    back = lib.Domain(**{k: pinned(torch.empty_like(getattr(st, k))) for k in NODE + ELEM})
    clock = lib.Scalars(0.0, st.dt, 1e20, 1e20, 0)
    return dict(case=case, ctx=ctx, start=start, back=back, clock=clock)


# ---- one pass -------------------------------------------------------------

def domain_out(dom):
    return {**{k: getattr(dom, k) for k in NODE + ELEM}, "time": float(dom.time), "deltatime": float(dom.deltatime)}


def run(state):
    case, lib = state["case"], package()
    if case["kind"] == "batch":
        with lib.Batch(state["sizes"], state["factors"], LULESH2, ORDER[case["prec"]]) as b:
            b.run(case["cycles"])
            out = {k: np.concatenate([b.get_field(i, k) for i in range(b.n)]) for k in ("x", "y", "z", "xd", "e", "p", "v")}
            ends = [b.instance(i) for i in range(b.n)]
        return dict(out, time=np.array([sc.time for sc, _, _ in ends]), cycle=np.array([sc.cycle for sc, _, _ in ends]),
                    origin=np.array([e for _, e, _ in ends]))
    ctx = state["ctx"]
    if case["kind"] == "step":
        ctx.scalars = state["clock"]
        return domain_out(lib.lulesh(ctx, state["start"]))
    ctx.upload(state["start"])
    ctx.scalars = state["clock"]
    if case["kind"] == "run":
        n = ctx.run(case["cycles"])
        return dict(domain_out(ctx.download(state["back"])), cycle=n)
    ctx.time_increment()
    ctx.lagrange_nodal()
    ctx.lagrange_elements()
    ctx.calc_time_constraints()
    sc = ctx.scalars
    return dict(domain_out(ctx.download(state["back"])), vdov=ctx.get_field("vdov"), arealg=ctx.get_field("arealg"),
                dtcourant=sc.dtcourant, dthydro=sc.dthydro)


# ---- what a pass cannot do without ----------------------------------------

# cycles of a problem that runs to its stop time, about
def cycles_of(case, s):
    if case["kind"] in ("step", "phases"):
        return 1
    return case["cycles"] or int(31 * s ** 1.0 if case.get("init") != LULESH1 else 59 * s)


def work(case):
    """Bytes: the evolving state read and written once a cycle with the masses and volumes (and, on a mesh given by
    lists, the lists) read, and the state's way up and down where the call takes it there.  Flops: the step's
    arithmetic in IEEE FP64, about 1500 per zone and cycle (the equation of state, 200 of them, again for each
    repetition that a region asks for)."""
    sizes = [int(k) for k in case["sizes"].split(",")] if case["kind"] == "batch" else [case["s"]]
    reps = 4.6 if case.get("regions") else 1.0
    total, flops = 0.0, 0.0
    for s in sizes:
        ne, nn, n = s ** 3, (s + 1) ** 3, cycles_of(case, s)
        total += n * (nn * 8 * (2 * 6 + 1) + ne * 8 * (2 * 5 + 2) + (ne * 56 if case.get("mesh") == "lists" else 0))
        total += 8 * (6 * nn + 5 * ne) * (1 if case["kind"] == "batch" else 2)
        flops += n * ne * (1300 + 200 * reps)
    return {"bytes": total, "flops": flops}


# ---- the step in plain 64-bit torch ----------------------------------------

SIGNS = torch.tensor([[-1, 1, 1, -1, -1, 1, 1, -1], [-1, -1, 1, 1, -1, -1, 1, 1], [-1, -1, -1, -1, 1, 1, 1, 1]],
                     dtype=torch.float64)


def cross(a, b):
    return torch.linalg.cross(a, b, dim=0)


def dot(a, b):
    return (a * b).sum(0)


def node_normals(c):
    """Each face's area vector, a quarter to each of its corners: [3, 8, elements]."""
    out = torch.zeros_like(c)
    for f in ((0, 1, 2, 3), (0, 4, 5, 1), (1, 5, 6, 2), (2, 6, 7, 3), (3, 7, 4, 0), (4, 7, 6, 5)):
        a, b, d, e = (c[:, i] for i in f)
        out[:, list(f)] += 0.25 * cross(0.5 * (e + d - b - a), 0.5 * (d + b - e - a))[:, None]
    return out


def step64(st, c, case, lim):
    """One cycle on the State's tensors; c: mesh lists and masses; lim: the constraints, updated."""
    if st.cycle:
        new = 1e20
        if lim["courant"] < new:
            new = lim["courant"] / 2
        if lim["hydro"] < new:
            new = lim["hydro"] * 2 / 3
        ratio = new / st.dt
        if ratio >= 1:
            new = st.dt if ratio < 1.1 else st.dt * 1.2 if ratio > 1.2 else new
        st.dt = min(new, 1e-2)
    target = 1e-2 - st.time
    if st.dt < target < 4 * st.dt / 3:
        target = 2 * st.dt / 3
    st.dt = min(st.dt, target)
    st.time += st.dt
    st.cycle += 1
    dt, nl = st.dt, st.nodes
    sg = SIGNS.to(nl.device)
    gam = torch.stack([sg[1] * sg[2], sg[0] * sg[2], sg[0] * sg[1], sg[0] * sg[1] * sg[2]])
    # forces: stress on the node normals and the hourglass control
    pos, vel = torch.stack([st.x, st.y, st.z]), torch.stack([st.xd, st.yd, st.zd])
    cx, cu = pos[:, nl], vel[:, nl]
    f = (st.p + st.q) * node_normals(cx)
    with torch.enable_grad():
        g = cx.clone().requires_grad_(True)
        dvdx, = torch.autograd.grad(hex_volume(g).sum(), g)
    determ = c["vol0"] * st.v
    hour = torch.einsum("mk,dkn->dmn", gam, cx)
    hg = gam[:, :, None] - torch.einsum("dkn,dmn->mkn", dvdx, hour) / determ
    coef = -3.0 * 0.01 * st.ss * c["mass"] / determ ** (1 / 3)
    f += coef * torch.einsum("mkn,dmn->dkn", hg, torch.einsum("mkn,dkn->dmn", hg, cu))
    force = torch.zeros_like(pos).index_add_(1, nl.reshape(-1), f.reshape(3, -1))
    acc = torch.where(st.symm, torch.zeros_like(pos), force / c["nmass"])
    vel = vel + acc * dt
    vel = torch.where(vel.abs() < 1e-7, torch.zeros_like(vel), vel)
    pos = pos + vel * dt
    # kinematics
    cx, cu = pos[:, nl], vel[:, nl]
    vol = hex_volume(cx)
    vnew = vol / c["vol0"]
    delv = vnew - st.v
    area = None
    for a, b, d, e in ((0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7)):
        u, w = cx[:, d] - cx[:, a], cx[:, e] - cx[:, b]
        k = 4 * dot(cross(u, w), cross(u, w))
        area = k if area is None else torch.maximum(area, k)
    length = 4 * vol / area.sqrt()
    half = torch.einsum("ik,dkn->idn", sg, cx - 0.5 * dt * cu)
    um = torch.einsum("ik,dkn->idn", sg, cu)
    cof = [cross(half[1], half[2]), cross(half[2], half[0]), cross(half[0], half[1])]
    vdov = sum(dot(cof[i], um[i]) for i in range(3)) / dot(half[0], cof[0])
    # monotonic viscosity
    m, tiny = torch.einsum("ik,dkn->idn", sg, cx) / 4, 1e-36
    volq = c["vol0"] * vnew
    phi, dvx = [], []
    for d in range(3):
        a = cross(m[(d + 1) % 3], m[(d + 2) % 3])
        delx = volq / (dot(a, a) + tiny).sqrt()
        dv = dot(a, um[d] / 4) / (volq + tiny)
        lo, hi = dv[c["nb"][2 * d]], dv[c["nb"][2 * d + 1]]
        if c["free"]:   # the cube's far faces: no slope beyond them
            hi = torch.where(c["nb"][2 * d + 1] == c["self"], torch.zeros_like(hi), hi)
        norm = 1 / (dv + tiny)
        lo, hi = lo * norm, hi * norm
        phi.append(torch.minimum(torch.minimum(0.5 * (lo + hi), 2 * lo), 2 * hi).clamp(0, 1))
        dvx.append((dv * delx).clamp(max=0))
    rho = c["mass"] / (c["vol0"] * vnew)
    there = vdov <= 0
    ql = torch.where(there, -0.5 * rho * sum(a * (1 - b) for a, b in zip(dvx, phi)), 0.0)
    qq = torch.where(there, (2.0 / 3.0) * rho * sum(a * a * (1 - b * b) for a, b in zip(dvx, phi)), 0.0)
    # equation of state
    vc = vnew.clamp(1e-9, 1e9)
    comp, half_v = 1 / vc - 1, vc - 0.5 * delv
    comp_half = torch.where(vc <= 1e-9, comp, 1 / half_v - 1)
    top = vc >= 1e9
    p_old = torch.where(top, 0.0, st.p)
    comp, comp_half = torch.where(top, 0.0, comp), torch.where(top, 0.0, comp_half)

    def pressure(e, k):
        b = (2.0 / 3.0) * (k + 1)
        p = b * e
        return b, torch.where((p.abs() < 1e-7) | top, 0.0, p).clamp(min=0)

    def sound(e, v2, b, p):
        k = (2.0 / 3.0) * e + v2 * v2 * b * p
        return torch.where(k <= .111111e-36, .333333e-18, k.clamp(min=0).sqrt())

    grow = delv > 0
    e = (st.e - 0.5 * delv * (p_old + st.q)).clamp(min=-1e15)
    b, ph = pressure(e, comp_half)
    vhalf = 1 / (1 + comp_half)
    q = torch.where(grow, 0.0, sound(e, vhalf, b, ph) * ql + qq)
    e = e + 0.5 * delv * (3 * (p_old + st.q) - 4 * (ph + q))
    e = torch.where(e.abs() < 1e-7, 0.0, e).clamp(min=-1e15)
    b, p = pressure(e, comp)
    qt = torch.where(grow, 0.0, sound(e, vc, b, p) * ql + qq)
    e = e - (7 * (p_old + st.q) - 8 * (ph + q) + (p + qt)) * delv / 6
    e = torch.where(e.abs() < 1e-7, 0.0, e).clamp(min=-1e15)
    b, p = pressure(e, comp)
    ss = sound(e, vc, b, p)
    qn = ss * ql + qq
    q = torch.where(grow, q, torch.where(qn.abs() < 1e-7, 0.0, qn))
    st.e, st.p, st.q, st.ss = e, p, q, ss
    st.v = torch.where((vnew - 1).abs() < 1e-10, 1.0, vnew)
    st.x, st.y, st.z = pos
    st.xd, st.yd, st.zd = vel
    st.vdov, st.arealg = vdov, length
    # time constraints
    live = vdov != 0
    dtf = ss * ss + torch.where(vdov < 0, 256.0 * length * length * vdov * vdov, 0.0)
    for key, val in (("courant", length / dtf.sqrt()), ("hydro", 0.1 / (vdov.abs() + 1e-20))):
        least = float(torch.where(live, val, 1e20).min())
        if least < 1e20:
            lim[key] = least


def exact(case, seed):
    if case["kind"] == "batch":
        return None   # hundreds of cycles of each instance: over the time that is worth spending here
    with torch.no_grad():
        st = State(case, seed)
        st.time, s = 0.0, case["s"]
        nb = torch.from_numpy(neighbours(s, case, seed)).to(st.x.device)
        nmass = torch.zeros_like(st.x).index_add_(0, st.nodes.reshape(-1), (st.vol0 / 8).repeat(8))
        c = dict(vol0=st.vol0, mass=st.vol0, nmass=nmass, nb=nb, free=case.get("mesh") != "lists",
                 self=torch.arange(s ** 3, device=st.x.device))
        lim, most = dict(courant=1e20, hydro=1e20), cycles_of(case, s)
        while st.time < 1e-2 and (case.get("cycles") == 0 or st.cycle < most):
            step64(st, c, case, lim)
        out = {**{k: getattr(st, k) for k in NODE + ELEM}, "time": st.time, "deltatime": st.dt}
    if case["kind"] == "run":
        out["cycle"] = None
    if case["kind"] == "phases":
        out.update(vdov=st.vdov, arealg=st.arealg, dtcourant=lim["courant"], dthydro=lim["hydro"])
    return out
