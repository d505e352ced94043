"""Performance cases of the LBM-PSM library: what its users have it do, each
pass through the public Python entry points (``lbmpsm.Lattice``, ``Ensemble``,
``Group``), with an independent 64-bit restatement of every pass in plain
torch (``exact``).

Kinds of a case
  step      coupling steps with moving particles, the DEM host's timestep loop:
            ``Lattice.step`` with host arrays or ``Lattice.step_device`` with
            device arrays, then ``Lattice.apply_bc`` where walls are set
  fixed     ``Lattice.run_fixed``: many steps past particles held in place,
            then the forces (verification decks, drag and permeability runs)
  group     ``Group.run_fixed`` over ensembles of boxes of several sizes, then
            the forces of every ensemble (parameter studies, training data)
  fields    a step whose density, velocity and solid fraction fields are read
            for output (``fix lbm-psm-vti``)
  restart   state in, one step, state out (``fix lbm-psm-restart``)
  adjoint   ``Lattice.adjoint_drag``: the drag's gradient
  tangent   ``Lattice.tangent_drag``: its derivative along a direction
Lattice units throughout: spacing, time step and density 1.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "lammps-lbm-psm_gb300"))
import lbmpsm  # noqa: E402
from lbmpsm.host import Domain, ghost_images  # noqa: E402

U_LB = 0.01  # characteristic lattice velocity: wall and inflow speed
LOOP = 16    # steps of the closed loop that every moving particle walks
AMP = 0.1    # its radius
WARM = 6     # steps before a field output
SHIFT = 0.3  # how far a seed moves a particle from its place

PERIODIC = {"none": (1, 1, 1), "shear": (1, 0, 1), "channel": (1, 0, 1), "xFlow": (0, 0, 0),
            "channel-velIn-pressOut": (0, 0, 0), "closedBox": (0, 0, 0)}


def _case(name, kind, n, storage, bc="none", particles=1, diam=12.0, tau=0.65, fx=0.0, steps=1, api="host", spin=False):
    return {"name": name, "kind": kind, "nx": n[0], "ny": n[1], "nz": n[2] if len(n) == 3 else 1, "dim": len(n),
            "storage": storage, "bc": bc, "particles": particles, "diam": diam, "tau": tau, "fx": fx, "steps": steps,
            "api": api, "spin": spin}


def listed():
    return [
        # one disc in a small periodic 2-D box, a step per call: the smallest
        # deck of all, where the call itself is what it costs
        _case("disc-2d-256-fp64", "step", (256, 256), "fp64", particles=1, diam=16.0, fx=1e-6),
        # a 2-D channel between walls with inflow and outflow, long ragged
        # rows, a few dozen spinning discs of a DEM run
        _case("channel-2d-601x187-fp32", "step", (601, 187), "fp32", bc="channel-velIn-pressOut", particles=24,
              diam=14.0, tau=0.7, steps=2, spin=True),
        # a fixed sphere in a periodic 3-D box driven by a body force: the
        # drag deck, hundreds of steps in a row without the host
        _case("sphere-128-fp32", "fixed", (128, 128, 128), "fp32", particles=1, diam=16.0, tau=0.7, fx=1e-6, steps=20),
        # the sheared dense suspension of the benchmark on device arrays, at
        # its full size: the largest everyday run
        _case("suspension-256-fp32", "step", (256, 256, 256), "fp32", bc="shear", particles=2000, steps=2, api="device"),
        # the same flow in a smaller ragged box, 16-bit storage, host arrays
        _case("suspension-190x150x222-fp16", "step", (190, 150, 222), "fp16", bc="shear", particles=700, steps=2),
        # the default precision (the reference's arithmetic) with spinning spheres
        _case("suspension-128x96x160-fp64", "step", (128, 96, 160), "fp64", bc="shear", particles=230, steps=2, spin=True),
        # a long duct: x-rows of 500 nodes, walls in y
        _case("duct-500x120x96-fp32", "step", (500, 120, 96), "fp32", bc="channel", particles=650, tau=0.8, fx=1e-6,
              steps=2, api="device"),
        # boxes of three edges, a parameter study stepped as one group
        _case("group-32-48-64-fp32", "group", (32, 48, 64), "fp32", particles=72, diam=11.0, steps=8),
        # field output of a wall-bounded 3-D flow
        _case("fields-160x90x120-fp32", "fields", (160, 90, 120), "fp32", bc="channel", particles=150, tau=0.7, fx=1e-6),
        # restart of an FP64 run
        _case("restart-96x80x70-fp64", "restart", (96, 80, 70), "fp64", bc="shear", particles=40),
        # gradient of the drag of a few spheres with respect to their places,
        # the viscosity and the driving force
        _case("adjoint-56-fp64", "adjoint", (56, 56, 56), "fp64", particles=8, diam=12.0, tau=0.7, fx=1e-5, steps=24),
        # its forward-mode counterpart
        _case("tangent-48-fp64", "tangent", (48, 48, 48), "fp64", particles=4, diam=12.0, tau=0.7, fx=1e-5, steps=16),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "fixed", "group", "fields", "restart", "adjoint", "tangent"])
    storage = "fp64" if kind in ("adjoint", "tangent") else rng.choice(["fp64", "fp32", "fp32", "fp16", "bf16"])
    tau = round(rng.uniform(0.6, 0.9), 3)
    if kind in ("adjoint", "tangent"):
        e = [_logint(rng, 34, 56) for _ in range(3)]
        return _case("", kind, e, "fp64", particles=rng.randint(1, 5), diam=round(rng.uniform(7.0, 13.0), 2), tau=tau,
                     fx=1e-5, steps=rng.randint(6, 24))
    if kind == "group":
        e = sorted(rng.sample(range(28, 72), 3))
        return _case("", kind, e, storage if storage != "fp64" else "fp32", particles=rng.randint(6, 60),
                     diam=round(rng.uniform(8.0, 12.0), 2), tau=tau, steps=8)
    dim = 2 if kind in ("step", "fixed") and rng.random() < 0.3 else 3
    bc = "none" if kind == "fixed" else rng.choice(["none", "shear", "channel", "closedBox", "channel-velIn-pressOut"])
    most = {"fp64": 2.0e6}.get(storage, 1.2e7 if kind in ("step", "fixed") else 2.0e6)
    nodes = math.exp(rng.uniform(math.log(4.0e4), math.log(most if dim == 3 else most / 4)))
    stretch = [math.exp(rng.uniform(-0.6, 0.6)) for _ in range(dim)]
    scale = (nodes / math.prod(stretch)) ** (1.0 / dim)
    n = [max(36, int(round(scale * s))) for s in stretch]
    while math.prod(n) > most:
        n[n.index(max(n))] = int(max(n) * 0.9)
    diam = round(rng.uniform(7.0, 16.0), 2)
    room = math.prod(max(m - diam - 4.0, 1.0) for m in n) / (diam ** dim * (0.7854 if dim == 2 else 0.5236))
    particles = max(1, min(2000, int(room * rng.uniform(0.01, 0.1))))
    return _case("", kind, n, storage, bc=bc, particles=1 if kind == "fixed" and rng.random() < 0.5 else particles,
                 diam=diam, tau=tau, fx=1e-6 if bc in ("none", "channel") else 0.0,
                 steps={"step": 2, "fixed": 10}.get(kind, 1), api=rng.choice(["host", "device"]) if kind == "step" else "host",
                 spin=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _periodic(case):
    p = PERIODIC[case["bc"]]
    return p if case["dim"] == 3 else (p[0], p[1], 1)


def _params(n, dim, periodic, tau, fx, diam):
    """The arguments of Lattice for n nodes per axis in lattice units."""
    nlc = int(diam) + 1
    nu = (tau - 0.5) / 3.0
    prd = tuple(1.0 if d >= dim else float(n[d] if periodic[d] else n[d] - 1) for d in range(3))
    return dict(dimension=dim, boxlo=(0.0, 0.0, 0.0), prd=prd, periodic=periodic, nevery=1, Nlc=nlc, lc=float(nlc - 1),
                rho=1.0, nu=nu, Re=U_LB * (nlc - 1) / nu, tau=tau, Fext=(fx, 0.0, 0.0))


def _place(rng, count, r, prm, gap):
    """Centres of up to `count` spheres of radius r, at least `gap` apart."""
    dim, L = prm["dimension"], np.array(prm["prd"])
    per = np.array([bool(p) for p in prm["periodic"]])
    lo, hi = np.where(per, 0.0, r + 2.0), np.where(per, L, L - r - 2.0)
    hi = np.maximum(hi, lo + 1e-3)
    c = np.zeros((count, 3))
    k = 0
    for _ in range(40 * count + 200):
        if k == count:
            break
        p = rng.uniform(lo, hi)
        if dim == 2:
            p[2] = 0.0
        if k:
            d = c[:k] - p
            d -= np.where(per, L * np.round(d / L), 0.0)
            if np.min(np.einsum("ij,ij->i", d[:, :dim], d[:, :dim])) < (2 * r + gap) ** 2:
                continue
        c[k] = p
        k += 1
    return c[:k]


def _images(layout, rng, prm, count, diam, moving, spin, gap=0.0):
    """Particle images (owned, then ghosts) on LOOP sets of positions: dict of
    tag[n], x[LOOP, n, 3], v[LOOP, n, 3], omega[n, 3], radius[n].  The layout
    is the case's own, so that every seed has as many images; the seed moves
    each particle within its gap and gives it its loop and spin."""
    dim, r = prm["dimension"], diam / 2
    x = _place(layout, count, r, prm, gap + 2 * SHIFT)
    m = len(x)
    omega = rng.normal(0.0, 2e-3, (m, 3)) if spin else np.zeros((m, 3))
    if dim == 2:
        omega[:, :2] = 0.0
    hi = tuple(prm["prd"])
    g = ghost_images(Domain(dim, (0.0, 0.0, 0.0), hi, prm["periodic"]), r + 3.0, np.arange(1, m + 1), x,
                     np.zeros((m, 3)), omega, np.full(m, r))
    src = np.asarray(g.owner).copy()
    for _ in range(4):
        src = np.where(src >= m, np.asarray(g.owner)[src], src)
    a, b = rng.normal(size=(m, 3)), rng.normal(size=(m, 3))
    if dim == 2:
        a[:, 2] = b[:, 2] = 0.0
    a /= np.linalg.norm(a, axis=1, keepdims=True)
    b /= np.linalg.norm(b, axis=1, keepdims=True)
    t = 2 * np.pi * np.arange(LOOP + 1)[:, None, None] / LOOP + rng.uniform(0.0, 2 * np.pi, (1, m, 1))
    d = (AMP if moving else 0.0) * (np.cos(t) * a + np.sin(t) * b)
    d = d + rng.uniform(-1.0, 1.0, (1, m, 3)) * ([SHIFT / math.sqrt(dim)] * dim + [0.0] * (3 - dim))
    return dict(tag=np.asarray(g.tag, np.int32), x=np.ascontiguousarray(np.asarray(g.x)[None] + d[:LOOP, src]),
                v=np.ascontiguousarray((d[1:] - d[:-1])[:, src]), omega=np.ascontiguousarray(g.omega, np.float64),
                radius=np.ascontiguousarray(g.radius, np.float64))


def _inputs(case, seed):
    """Lattice arguments and particle images of a case of one lattice."""
    rng, layout = np.random.default_rng([int(seed), 11]), np.random.default_rng([case["nx"], case["ny"], case["nz"], 13])
    n = (case["nx"], case["ny"], case["nz"])
    grad = case["kind"] in ("adjoint", "tangent")
    prm = _params(n, case["dim"], _periodic(case), case["tau"], case["fx"], case["diam"])
    moving = not grad and case["kind"] != "fixed"
    img = _images(layout, rng, prm, case["particles"], case["diam"], moving, case["spin"], gap=4.0 if grad else 0.0)
    return prm, img, rng


def _group_inputs(case, seed):
    """Per edge class: the boxes' arguments and their images with box indices."""
    rng, layout = np.random.default_rng([int(seed), 12]), np.random.default_rng([case["nx"], case["ny"], case["nz"], 14])
    classes = []
    for e, share in zip((case["nx"], case["ny"], case["nz"]), (0.5, 0.3, 0.2)):
        boxes, cols = [], []
        for b in range(max(1, int(round(case["particles"] * share)))):
            tau, fx = round(float(rng.uniform(0.6, 1.0)), 4), float(rng.uniform(1e-7, 1e-5))
            boxes.append(_params((e, e, e), 3, (1, 1, 1), tau, fx, 12.0))
            img = _images(layout, rng, boxes[-1], int(layout.integers(1, 6)), case["diam"], False, False)
            cols.append(dict(box=np.full(len(img["tag"]), b, np.int32), tag=img["tag"], x=img["x"][0], v=img["v"][0],
                             omega=img["omega"], radius=img["radius"]))
        classes.append((boxes, {k: np.concatenate([c[k] for c in cols]) for k in cols[0]}))
    return classes


def _restart_state(rng, local, dim):
    """Populations of a slowly varying flow, in the library's exchange layout."""
    E, w = _set(dim)
    ax = [torch.arange(m, dtype=torch.float64, device="cuda") * (2 * math.pi / max(m - 2, 1)) for m in local]
    g = torch.meshgrid(*ax, indexing="ij")
    ph = rng.uniform(0.0, 2 * math.pi, (4, 3))
    wave = [torch.sin(g[0] + ph[c, 0]) * torch.cos(g[1] + ph[c, 1]) * torch.cos(g[2] + ph[c, 2]) for c in range(4)]
    rho, u = 1.0 + 2e-3 * wave[0], [U_LB * wave[1 + c] for c in range(3)]
    if dim == 2:
        u[2] = torch.zeros_like(u[2])
    uu = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    f = torch.stack([w[q] * rho * (1 + 3 * eu + 4.5 * eu ** 2 - 1.5 * uu)
                     for q in range(len(w)) for eu in [E[q][0] * u[0] + E[q][1] * u[1] + E[q][2] * u[2]]], dim=-1)
    return f.cpu().numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "group":
        ens, ns = [], []
        for boxes, img in _group_inputs(case, seed):
            e = lbmpsm.Ensemble(boxes, storage=case["storage"])
            e.step(img["box"], img["tag"], img["x"], img["v"], img["omega"], img["radius"])
            ens.append(e)
            ns.append(len(img["tag"]))
        return {"kind": kind, "group": lbmpsm.Group(ens), "members": ens, "n": ns, "steps": case["steps"]}
    prm, img, rng = _inputs(case, seed)
    n = len(img["tag"])
    lat = lbmpsm.Lattice(**prm, storage=case["storage"], max_images=n, max_radius=case["diam"] / 2)
    if case["bc"] != "none":
        lat.set_bc(case["bc"])
    s = {"kind": kind, "lat": lat, "img": img, "n": n, "steps": case["steps"], "bc": case["bc"] != "none", "k": 0,
         "api": case["api"]}
    if kind == "fixed":
        lat.step(img["tag"], img["x"][0], img["v"][0], img["omega"], img["radius"])
    elif case["api"] == "device":
        s["dev"] = {k: torch.as_tensor(v, device="cuda") for k, v in img.items()}
        s["out"] = torch.zeros((case["steps"], 12 * n), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()  # the library works on a stream of its own
    else:
        s["out"] = np.zeros((case["steps"], 12 * n))
    if kind == "restart":
        s["f"] = _restart_state(rng, lat.local, case["dim"])
    if kind == "tangent":
        s["dx"] = rng.normal(size=(n, 3))
    if kind == "fields":  # a flow that has begun
        for j in range(WARM):
            lat.step(img["tag"], img["x"][j], img["v"][j], img["omega"], img["radius"])
            lat.apply_bc()
        s["k"] = WARM
    return s


def run(state):
    kind, steps = state["kind"], state["steps"]
    if kind == "group":
        state["group"].run_fixed(steps)
        return [m.read_forces(n) for m, n in zip(state["members"], state["n"])]
    lat, img = state["lat"], state["img"]
    if kind == "fixed":
        lat.run_fixed(steps)
        return lat.read_forces(state["n"])
    if kind == "adjoint":
        return lat.adjoint_drag(img["tag"], img["x"][0], img["v"][0], img["omega"], img["radius"], steps, steps // 2, steps,
                                checkpoint_every=max(1, int(math.sqrt(steps))))
    if kind == "tangent":
        return lat.tangent_drag(img["tag"], img["x"][0], img["v"][0], img["omega"], img["radius"], steps, steps // 2, steps,
                                dtau=0.3, dFext=(1e-6, 2e-6, -1e-6), dx=state["dx"])
    if kind == "restart":
        lat.set_populations(state["f"])
    if kind == "fields":
        lat.request_macro()
    for s in range(steps):
        j = state["k"] % LOOP
        state["k"] += 1
        if state["api"] == "device":
            d, o, n = state["dev"], state["out"][s], state["n"]
            lat.step_device(n, d["tag"].data_ptr(), d["x"][j].data_ptr(), d["v"][j].data_ptr(), d["omega"].data_ptr(),
                            d["radius"].data_ptr(), o.data_ptr(), o.data_ptr() + 24 * n, o.data_ptr() + 48 * n)
        else:
            lat.step(img["tag"], img["x"][j], img["v"][j], img["omega"], img["radius"], out=state["out"][s])
        if state["bc"]:
            lat.apply_bc()
    if kind == "fields":
        return {"forces": state["out"], "fields": lat.export_fields(as_double=False)}
    if kind == "restart":
        return {"forces": state["out"], "f": lat.populations()}
    return state["out"]


BYTES = {"fp64": 8, "fp32": 4, "fp16": 2, "bf16": 2}


def work(case):
    """Every population read and written once a step (the sweeps: forward, and
    the reverse's state and adjoint), image arrays and outputs once."""
    q = 9 if case["dim"] == 2 else 19
    flops = 140.0 if q == 9 else 300.0  # macroscopic values, equilibrium and relaxation of a node
    kind, steps = case["kind"], case["steps"]
    nodes = case["nx"] * case["ny"] * case["nz"]
    if kind == "group":
        nodes = sum(max(1, int(round(case["particles"] * s))) * e ** 3
                    for e, s in zip((case["nx"], case["ny"], case["nz"]), (0.5, 0.3, 0.2)))
    b = 2.0 * q * BYTES[case["storage"]] * nodes * steps + 180.0 * case["particles"] * steps
    f = flops * nodes * steps
    if kind == "adjoint":
        b, f = b * 2.5, f * 2.5
    elif kind == "tangent":
        b, f = b * 2.0, f * 2.5
    elif kind == "fields":
        b += 20.0 * nodes
    elif kind == "restart":
        b += 16.0 * q * nodes
    return {"bytes": b, "flops": f}


# ------------------------------------------------------- 64-bit restatement
E19 = [(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, -1, 0), (1, 0, 1),
       (-1, 0, -1), (0, 1, 1), (0, -1, -1), (1, -1, 0), (-1, 1, 0), (1, 0, -1), (-1, 0, 1), (0, 1, -1), (0, -1, 1)]
E9 = [(0, 0, 0), (1, 0, 0), (0, 1, 0), (-1, 0, 0), (0, -1, 0), (1, 1, 0), (-1, 1, 0), (-1, -1, 0), (1, -1, 0)]


def _set(dim):
    if dim == 2:
        return E9, [4 / 9] + [1 / 9] * 4 + [1 / 36] * 4
    return E19, [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12


class _Flow:
    """One lattice in FP64: populations f[q] on the stored nodes (periodic axes
    the interior nodes, other axes also the halo planes), the two-slot particle
    table and the coupling step."""

    def __init__(self, prm, bc="none"):
        self.dim = dim = prm["dimension"]
        self.E, self.w = _set(dim)
        self.per = [d >= dim or bool(prm["periodic"][d]) for d in range(3)]
        n = [int(prm["prd"][d] + 1.5) - (1 if prm["periodic"][d] else 0) if d < dim else 1 for d in range(3)]
        self.L = [n[d] + 2 if d < dim else 1 for d in range(3)]
        self.off = [1 if d < dim and self.per[d] else 0 for d in range(3)]
        self.S = [n[d] if d >= dim or self.per[d] else n[d] + 2 for d in range(3)]
        self.tau, self.bc = prm["tau"], bc
        self.F = [float(v) for v in prm["Fext"]]
        kw = dict(dtype=torch.float64, device="cuda")
        self.f = torch.stack([torch.full(self.S, w, **kw) for w in self.w])
        self.id = [torch.zeros(self.S, dtype=torch.int32, device="cuda") for _ in range(2)]
        self.eps = [torch.zeros(self.S, **kw) for _ in range(2)]
        self.us = [torch.zeros([3] + self.S, **kw) for _ in range(2)]
        self.nf = [torch.zeros([3] + self.S, **kw) for _ in range(2)]

    def _axes(self, lo, hi):
        return [torch.arange(lo[d], hi[d], dtype=torch.float64, device="cuda").reshape([-1 if a == d else 1 for a in range(3)])
                for d in range(3)]

    def _solid(self, lo, hi, xl, r):
        """Solid fraction of nodes [lo, hi): sub-cell centres inside the sphere."""
        dim = self.dim
        D = [a - xl[d] for d, a in enumerate(self._axes(lo, hi))]
        dist = D[0] ** 2 + D[1] ** 2 + D[2] ** 2
        h = math.sqrt(3.1 if dim == 3 else 2.1) / 2
        sub = (torch.arange(10, dtype=torch.float64, device="cuda") + 0.5) * 0.1 - 0.5
        sq = [(D[d].unsqueeze(-1) + sub) ** 2 for d in range(dim)]
        s = sq[0].unsqueeze(-1) + sq[1].unsqueeze(-2)
        if dim == 2:
            cnt = (s < r * r).sum((-1, -2)).double() / 100.0
        else:
            cnt = (s.unsqueeze(-1) + sq[2].unsqueeze(-2).unsqueeze(-2) < r * r).sum((-1, -2, -3)).double() / 1000.0
        e = torch.where(dist < (r - h) ** 2, torch.ones_like(dist), cnt)
        return torch.where(dist > (r + h) ** 2, torch.zeros_like(dist), e), D

    def _box(self, xl, r):
        lo, hi = [], []
        for d in range(3):
            a = min(max(int(xl[d] - r) - 2, 0), self.L[d])
            b = min(max(int(xl[d] + r) + 2, 0 if d < 2 else 1), self.L[d])
            if self.off[d]:
                a, b = max(a, 1), min(b, self.L[d] - 1)
            lo.append(a)
            hi.append(b)
        return lo, hi

    def _slice(self, lo, hi):
        return tuple(slice(lo[d] - self.off[d], hi[d] - self.off[d]) for d in range(3))

    def map(self, img):
        for t, x, v, om, r in zip(img["tag"].tolist(), img["x"].tolist(), img["v"].tolist(), img["omega"].tolist(),
                                  img["radius"].tolist()):
            xl = [c + 1.0 for c in x]
            lo, hi = self._box(xl, r)
            if any(a >= b for a, b in zip(lo, hi)):
                continue
            e, D = self._solid(lo, hi, xl, r)
            s = self._slice(lo, hi)
            i0, i1 = self.id[0][s], self.id[1][s]
            on = e > 1e-5
            m0 = i0 == t
            m1 = ~m0 & (i1 == t)
            set0 = on & (m0 | (~m1 & (i0 == 0)))
            set1 = on & ~set0 & (m1 | (i1 == 0))
            u = [v[0] + om[1] * D[2] - om[2] * D[1], v[1] + om[2] * D[0] - om[0] * D[2], v[2] + om[0] * D[1] - om[1] * D[0]]
            for k, put, gone in ((0, set0, ~on & m0), (1, set1, ~on & m1)):
                self.id[k][s] = torch.where(put, t, torch.where(gone, 0, self.id[k][s]))
                self.eps[k][s] = torch.where(put, e, torch.where(gone, 0.0, self.eps[k][s]))
                for c in range(3):
                    self.us[k][c][s] = torch.where(put, u[c] + torch.zeros_like(e), self.us[k][c][s])

    def collide(self):
        E, w, om, F, f = self.E, self.w, 1.0 / self.tau, self.F, self.f
        rho = f.sum(0)
        j = [sum(E[q][c] * f[q] for q in range(len(w)) if E[q][c]) + 0.5 * F[c] if c < self.dim else torch.zeros_like(rho)
             for c in range(3)]
        u = [c / rho for c in j]
        self.rho, self.u = rho, u
        uu = 1.5 * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
        at = torch.nonzero(((self.id[0] > 0) | (self.id[1] > 0)).reshape(-1)).reshape(-1)
        rp = rho.reshape(-1)[at]
        B = [self.eps[k].reshape(-1)[at] * (self.id[k].reshape(-1)[at] > 0) for k in range(2)]
        tot = torch.clamp(B[0] + B[1], min=1.0)
        B = [b / tot for b in B]
        us = [[self.us[k][c].reshape(-1)[at] for c in range(3)] for k in range(2)]
        uus = [1.5 * (a[0] ** 2 + a[1] ** 2 + a[2] ** 2) for a in us]
        acc = [[torch.zeros_like(rp) for _ in range(3)] for _ in range(2)]
        new = torch.empty_like(f)
        for q, (e, wq) in enumerate(zip(E, w)):
            eu = e[0] * u[0] + e[1] * u[1] + e[2] * u[2]
            feq = wq * rho * (1 + 3 * eu + 4.5 * eu * eu - uu)
            eF = e[0] * F[0] + e[1] * F[1] + e[2] * F[2]
            Fq = (1 - 0.5 * om) * wq * (3 * (eF - u[0] * F[0] - u[1] * F[1] - u[2] * F[2]) + 9 * eu * eF)
            out = f[q] + om * (feq - f[q]) + Fq
            if len(at):
                fp, fe = f[q].reshape(-1)[at], feq.reshape(-1)[at]
                g = fp + (1 - B[0] - B[1]) * om * (fe - fp) + Fq.reshape(-1)[at]
                for k in range(2):
                    es = e[0] * us[k][0] + e[1] * us[k][1] + e[2] * us[k][2]
                    t = B[k] * (wq * rp * (1 + 3 * es + 4.5 * es * es - uus[k]) - fp + (1 - om) * (fp - fe))
                    g = g + t
                    for c in range(3):
                        if e[c]:
                            acc[k][c] -= e[c] * t
                out.reshape(-1)[at] = g
            new[q] = torch.roll(out, e, (0, 1, 2))
            for d in range(3):
                if e[d] and not self.per[d]:  # nothing streams in from outside the array
                    new[q].select(d, 0 if e[d] > 0 else -1).fill_(wq)
        for k in range(2):
            self.nf[k].zero_()
            for c in range(3):
                self.nf[k][c].reshape(-1)[at] = acc[k][c]
        self.f = new

    def walls(self):
        """Zou-He closures of the selected keyword, face after face."""
        u, L, dim = U_LB, self.L, self.dim
        x0, x1, y0, y1 = (0, 1, "v"), (0, -1, "v"), (1, 1, "v"), (1, -1, "v")
        z = [(2, 1, "v"), (2, -1, "v")] if dim == 3 else []
        faces = {"none": [], "shear": [(y0, -u), (y1, u)], "channel": [(y0, 0.0), (y1, 0.0)],
                 "channel-velIn-pressOut": [(x0, u), ((0, -1, "d"), 1.0), (y0, 0.0), (y1, 0.0)] + [(a, 0.0) for a in z],
                 "closedBox": [(x0, 0.0), (x1, 0.0), (y0, 0.0), (y1, 0.0)] + [(a, 0.0) for a in z]}[self.bc]
        for (ax, s, what), p in faces:
            sl = []
            for d in range(3):
                if d >= dim:
                    sl.append(slice(0, 1))
                elif d == ax:
                    at = 1 if s > 0 else L[d] - 2
                    sl.append(slice(at, at + 1))
                else:
                    sl.append(slice(1 - self.off[d], L[d] - 1 - self.off[d]))
            g = self.f[(slice(None),) + tuple(sl)]
            E, Q = self.E, range(len(self.E))
            opp = [E.index(tuple(-c for c in e)) for e in E]
            total = sum(g[q] for q in Q if E[q][ax] == 0) + 2 * sum(g[q] for q in Q if E[q][ax] == -s)
            if what == "d":
                rho, un = p + torch.zeros_like(total), total / p - 1.0
            else:
                un = p if ax == 0 else 0.0
                rho = total / (1.0 - s * un)
            vel = [un, 0.0, 0.0] if ax == 0 else [p, 0.0, 0.0]
            N = [None if d == ax else 0.5 * (sum(g[q] for q in Q if E[q][ax] == 0 and E[q][d] == 1)
                                             - sum(g[q] for q in Q if E[q][ax] == 0 and E[q][d] == -1))
                 - (rho * vel[d] / 3 if dim == 3 else 0.5 * rho * vel[d] - rho * vel[d] / 6) for d in range(dim)]
            new = {}
            for q in Q:
                e = E[q]
                if e[ax] != s:
                    continue
                eu = sum(e[d] * vel[d] for d in range(3))
                side = [d for d in range(dim) if d != ax and e[d]]
                if side:
                    new[q] = g[opp[q]] + rho * eu / 6 - e[side[0]] * N[side[0]]
                else:
                    new[q] = g[opp[q]] + rho * eu * (1 / 3 if dim == 3 else 2 / 3)
            for q, v in new.items():
                g[q] = v

    def forces(self, img):
        """fh | th | S of every image, one row of 12n values."""
        fh, th, st = [], [], []
        for t, x, r in zip(img["tag"].tolist(), img["x"].tolist(), img["radius"].tolist()):
            xl = [c + 1.0 for c in x]
            lo, hi = self._reduce_box(xl, r)
            if any(a >= b for a, b in zip(lo, hi)):
                z = torch.zeros((), dtype=torch.float64, device="cuda")
                fh += [z] * 3
                th += [z] * 3
                st += [z] * 6
                continue
            s = self._slice(lo, hi)
            D = [a - xl[d] for d, a in enumerate(self._axes(lo, hi))]
            m0 = self.id[0][s] == t
            m1 = ~m0 & (self.id[1][s] == t)
            G = [torch.where(m0, self.nf[0][c][s], torch.where(m1, self.nf[1][c][s], 0.0)) for c in range(3)]
            P = [[(D[a] * G[b]).sum() for b in range(3)] for a in range(3)]
            fh += [g.sum() for g in G]
            th += [P[1][2] - P[2][1], P[2][0] - P[0][2], P[0][1] - P[1][0]]
            st += [-P[0][0], -P[1][1], -P[2][2], -0.5 * (P[1][0] + P[0][1]), -0.5 * (P[2][0] + P[0][2]),
                   -0.5 * (P[2][1] + P[1][2])]
        return torch.stack(fh), torch.stack(th), torch.stack(st)

    def _reduce_box(self, xl, r):
        lo, hi = [], []
        for d in range(3):
            a, b = int(xl[d] - r) - 2, int(xl[d] + r) + 2
            if d < self.dim:
                a, b = (min(max(c, 1), self.L[d] - 1) for c in (a, b))
            else:
                a, b = 0, 1
            lo.append(a)
            hi.append(b)
        return lo, hi

    def step(self, img):
        self.map(img)
        self.collide()
        return self.forces(img)


def _at(img, j):
    return dict(img, x=img["x"][j % LOOP], v=img["v"][j % LOOP])


def _exact_fixed(prm, img, steps):
    fl = _Flow(prm)
    fl.map(img)
    for _ in range(steps):
        fl.collide()
    return fl.forces(img)


def _exact_gradient(case, seed):
    """J, its gradient and the drag of every step, by reverse-mode
    differentiation of the whole run; the centre derivative of a node's solid
    fraction is the central difference of its sub-cell count."""
    prm, img, rng = _inputs(case, seed)
    T, fl, im = case["steps"], _Flow(prm), _at(img, 0)
    fl.map(im)
    if bool((fl.id[1] > 0).any()):
        return None
    E, w = fl.E, fl.w
    own, cw, us = fl.id[0].clone(), torch.zeros_like(fl.eps[0]), fl.us[0].clone()
    rows = list(zip(im["tag"].tolist(), im["x"].tolist(), im["v"].tolist(), im["radius"].tolist()))
    for t, x, v, r in rows:  # nodes next to a surface belong to its particle
        xl = [c + 1.0 for c in x]
        lo, hi = fl._box(xl, r)
        if any(a >= b for a, b in zip(lo, hi)):
            continue
        s, D = fl._slice(lo, hi), [a - xl[d] for d, a in enumerate(fl._axes(lo, hi))]
        own[s] = torch.where((own[s] == 0) & (D[0] ** 2 + D[1] ** 2 + D[2] ** 2 < (r + 1.5) ** 2), t, own[s])
    for t, x, v, r in rows:
        lo, hi = fl._reduce_box([c + 1.0 for c in x], r)
        if all(a < b for a, b in zip(lo, hi)):
            s = fl._slice(lo, hi)
            cw[s] += (own[s] == t).double()
    tau = torch.tensor(prm["tau"], dtype=torch.float64, device="cuda", requires_grad=True)
    F = torch.tensor(fl.F, dtype=torch.float64, device="cuda", requires_grad=True)
    eps = fl.eps[0].clone().requires_grad_(True)
    Et, wt = torch.tensor(E, dtype=torch.float64, device="cuda"), torch.tensor(w, dtype=torch.float64, device="cuda")
    col = wt.reshape(-1, 1, 1, 1)
    f, om, drags = fl.f, 1.0 / tau, []
    es = torch.tensordot(Et, us, 1)
    shape = col * (1 + 3 * es + 4.5 * es * es - 1.5 * (us * us).sum(0))
    del es
    for _ in range(T):
        rho = f.sum(0)
        m = torch.tensordot(Et.T, f, 1)
        u = (m + 0.5 * F.reshape(3, 1, 1, 1)) / rho
        eu = torch.tensordot(Et, u, 1)
        feq = col * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * (u * u).sum(0))
        eF = (Et @ F).reshape(-1, 1, 1, 1)
        Fq = (1 - 0.5 * om) * col * (3 * (eF - torch.tensordot(F, u, 1)) + 9 * eu * eF)
        so = shape * rho - f + (1 - om) * (f - feq)
        post = f + (1 - eps) * om * (feq - f) + eps * so + Fq
        drags.append(-(cw * eps * so[[q for q in range(len(E)) if E[q][0] == 1]].sum(0)).sum()
                     + (cw * eps * so[[q for q in range(len(E)) if E[q][0] == -1]].sum(0)).sum())
        f = torch.stack([torch.roll(post[q], E[q], (0, 1, 2)) for q in range(len(E))])
    t0 = T // 2
    J = sum(drags[t0 - 1:]) / (T - t0 + 1)
    dtau, dF, de = torch.autograd.grad(J, (tau, F, eps))
    h, dx = 1e-4, torch.zeros((len(rows), 3), dtype=torch.float64, device="cuda")
    for i, (t, x, v, r) in enumerate(rows):
        lo, hi = fl._box([c + 1.0 for c in x], r)
        if any(a >= b for a, b in zip(lo, hi)):
            continue
        s = fl._slice(lo, hi)
        mine = (own[s] == t).double() * de[s]
        for a in range(3):
            e = [fl._solid(lo, hi, [c + (g if d == a else 0.0) + 1.0 for d, c in enumerate(x)], r)[0] for g in (h, -h)]
            dx[i, a] = (mine * (e[0] - e[1]) / (2 * h)).sum()
    return dict(J=J.detach(), dtau=dtau, dFext=dF, dx=dx, drag=torch.stack(drags).detach()), rng


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "group":
        outs = []
        for boxes, img in _group_inputs(case, seed):
            per = []
            for b, prm in enumerate(boxes):
                mine = {k: v[img["box"] == b] for k, v in img.items()}
                per.append(_exact_fixed(prm, mine, steps + 1))
            outs.append(tuple(torch.cat([p[c] for p in per]) for c in range(3)))
        return outs
    if kind in ("adjoint", "tangent"):
        got = _exact_gradient(case, seed)
        if got is None:
            return None
        g, rng = got
        if kind == "adjoint":
            return g
        d = torch.tensor(rng.normal(size=tuple(g["dx"].shape)), dtype=torch.float64, device="cuda")
        v = 0.3 * g["dtau"] + (torch.tensor([1e-6, 2e-6, -1e-6], dtype=torch.float64, device="cuda") * g["dFext"]).sum()
        return g["J"], v + (g["dx"] * d).sum()
    prm, img, rng = _inputs(case, seed)
    if kind == "fixed":
        return _exact_fixed(prm, _at(img, 0), steps + 1)
    fl = _Flow(prm, case["bc"])
    if kind == "restart":
        f = torch.as_tensor(_restart_state(rng, fl.L, case["dim"]), device="cuda").movedim(-1, 0)
        f = f[(slice(None),) + tuple(slice(fl.off[d], fl.L[d] - fl.off[d]) for d in range(3))]
        for q, e in enumerate(fl.E):
            keep = torch.ones(fl.S, dtype=torch.bool, device="cuda")
            for d in range(3):
                if e[d] and not fl.per[d]:
                    keep.select(d, 0 if e[d] > 0 else -1).fill_(False)
            fl.f[q] = torch.where(keep, f[q], fl.f[q])
    out = []
    for s in range(steps + (WARM if kind == "fields" else 0)):
        out.append(torch.cat(fl.step(_at(img, s))))
        fl.walls()
    out = torch.stack(out[-steps:])
    if kind == "fields":
        s = tuple(slice(1 - fl.off[d], fl.L[d] - 1 - fl.off[d]) if d < fl.dim else slice(0, 1) for d in range(3))
        solid = torch.clamp(fl.eps[0] + fl.eps[1], max=1.0)
        flat = [a[s].permute(2, 1, 0).reshape(-1) for a in (solid, fl.rho, *fl.u)]
        return {"forces": out, "fields": (flat[0], flat[1], torch.stack(flat[2:], dim=-1))}
    if kind == "restart":
        f = fl.f
        for d in range(3):
            if fl.off[d]:  # halo planes of periodic axes are their twins
                f = torch.cat([f.narrow(d + 1, fl.S[d] - 1, 1), f, f.narrow(d + 1, 0, 1)], d + 1)
        return {"forces": out, "f": f.movedim(0, -1)}
    return out
