"""Cases on which the DEM step's speed is measured.

Each case is one call sequence of a program that uses the framework, over the
sizes of the configurations in pacific_b200/scenarios.py and of the tests:

* ``gas``     colliding spheres in a periodic box (few, short contacts): the
              leapfrog, the contact filter and the pair-list rebuild
* ``bed``     spheres packed in a walled box under gravity, about six lasting
              contacts each: the narrow phase, the force law and its memory
* ``batch``   a parameter sweep of independent packed boxes in one launch chain
* ``pour``    cubes, tetrahedra (and cylinders) falling: closest-point searches
* ``coupled`` a fluid solver's exchange: hydrodynamic forces in, a few
              sub-steps, positions and velocities out
* ``adjoint`` gradients of a trajectory loss for calibration (a forward run and
              the reverse sweep)

A pass of the first five runs ``steps`` leapfrog steps and reads the whole
state back into pinned host memory, as a program does at an output time; it
continues from the state that the previous pass left.
"""
from __future__ import annotations

import ctypes
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from pacific_b200 import FP32_SPLIT, FP64, Grains, library, scenarios
from pacific_b200.adjoint import Adjoint

P_TARGET = (2.0e4, 0.6, 0.35)       # kn, en, muc of the calibration target
P_START = (2.1e4, 0.57, 0.3675)     # and where the calibration starts


def listed():
    return [
        # A fluid solver with a few hundred resolved particles: the smallest
        # calls, where launches and synchronisations count (FP64, the coupling
        # library's default).
        dict(name="coupled_200_fp64", kind="coupled", n=200, precision="fp64", steps=4),
        # A laboratory box of 1,000 spheres between two outputs, FP64 as the
        # reference computes it.
        dict(name="bed_1000_fp64", kind="bed", n=1000, precision="fp64", steps=100,
             law="HookeMemory", mur=0.0),
        # The same size of study in FP32-split, without tangential memory and
        # with a ragged particle count.
        dict(name="bed_7777_hooke_fp32", kind="bed", n=7777, precision="fp32", steps=100,
             law="Hooke", mur=0.0),
        # A production bed in FP32-split, with rolling resistance.
        dict(name="bed_250k_fp32", kind="bed", n=250_000, precision="fp32", steps=100,
             law="HookeMemory", mur=0.02),
        # The same law at FP64.
        dict(name="bed_60k_fp64", kind="bed", n=60_000, precision="fp64", steps=100,
             law="HookeMemory", mur=0.0),
        # The 1M-sphere cooling gas: the largest single system, both modes
        # (FP64 at a quarter of it).
        dict(name="gas_1m_fp32", kind="gas", n=1_000_000, precision="fp32", steps=100),
        dict(name="gas_256k_fp64", kind="gas", n=256_000, precision="fp64", steps=100),
        # 200,000 cubes and tetrahedra, falling and colliding.
        dict(name="pour_200k_fp32", kind="pour", n=200_000, precision="fp32", steps=50, warm=200,
             cylinders=False),
        # A smaller pour with cylinders, FP64.
        dict(name="pour_20k_cyl_fp64", kind="pour", n=20_000, precision="fp64", steps=50, warm=200,
             cylinders=True),
        # A calibration sweep: 64 boxes of 500 to 20,000 spheres with their
        # own contact parameters, stepped together.
        dict(name="batch_64_fp32", kind="batch", n=64, nmax=20_000, precision="fp32", steps=50),
        # One gradient of the calibration loss at the configuration's size.
        dict(name="adjoint_4096", kind="adjoint", n=4096, steps=200, every=50),
        # And of a small one, whose every step is latency.
        dict(name="adjoint_200", kind="adjoint", n=200, steps=100, every=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("coupled", "bed", "bed", "bed", "gas", "gas", "pour", "batch", "adjoint"))
    prec = rng.choice(("fp32", "fp64"))
    if kind == "coupled":
        return dict(kind=kind, n=_log_int(rng, 50, 5000), precision=prec,
                    steps=rng.randint(1, 10))
    if kind == "bed":
        law = rng.choice(("HookeMemory", "HookeMemory", "Hooke"))
        return dict(kind=kind, n=_log_int(rng, 300, 250_000), precision=prec,
                    steps=rng.randint(20, 100), law=law,
                    mur=rng.choice((0.0, 0.02)) if law == "HookeMemory" else 0.0)
    if kind == "gas":
        return dict(kind=kind, n=_log_int(rng, 2000, 400_000), precision=prec,
                    steps=rng.randint(50, 100))
    if kind == "pour":
        return dict(kind=kind, n=_log_int(rng, 2000, 100_000), precision=prec,
                    steps=rng.randint(20, 50), warm=rng.randint(100, 200),
                    cylinders=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, n=rng.randint(4, 64), nmax=_log_int(rng, 1000, 20_000),
                    precision=prec, steps=rng.randint(20, 50))
    return dict(kind=kind, n=_log_int(rng, 150, 4096), steps=rng.randint(40, 150),
                every=rng.randint(10, 60))


# ------------------------------------------------------------------ scenes --
def _packed(n, seed, kn=1.0e4, en=0.7, muc=0.5, law="HookeMemory", mur=0.0, radius=1.0e-3):
    """A settled bed: spheres on a cubic lattice between six walls, each layer
    overlapping the one below by the weight it carries over kn and its lateral
    neighbours by 4e-7 m, slightly disturbed (overlaps by a few percent,
    velocities of 1e-4 m/s: the sliding of a creeping bed)."""
    side = max(2, round(n ** (1.0 / 3.0) / 1.26))        # a bed 2 times as high as wide
    layers = -(-n // (side * side))
    lateral = 2.0 * radius - 4.0e-7
    box = (lateral * (side + 1.0e-6), lateral * (side + 1.0e-6), lateral * (layers + 2.5))
    sc = scenarios.settling_box(n=n, seed=seed, box=box, radius=radius, spacing=lateral,
                                jitter=2.0e-9, vmax=1.0e-4, kn=kn, en=en, etat=None, muc=muc,
                                law=law, kr=0.01 if law == "Hooke" else 0.0)
    layer = np.arange(n) // (side * side)
    sag = sc.types[0]["density"] * 4.0 / 3.0 * math.pi * radius ** 3 * 9.81 / kn
    # overlap below layer k: the weight of the layers from k up
    z = radius + 2.0 * radius * np.arange(layers) - sag * np.cumsum(layers - np.arange(layers))
    sc.x[:, 2] += (z - lateral * (np.arange(layers) + 0.5))[layer]
    if mur:
        for m in sc.models:
            m["mur"] = mur
    return sc


def _scenes(case, seed):
    """The case's instances (one, except in a batch)."""
    kind = case["kind"]
    if kind in ("bed", "coupled"):
        return [_packed(case["n"], seed, law=case.get("law", "HookeMemory"),
                        mur=case.get("mur", 0.0))]
    if kind == "gas":
        n_fcc = math.ceil((case["n"] / 4.0) ** (1.0 / 3.0))
        return [scenarios.periodic_gas(n_fcc=n_fcc, n_target=case["n"], seed=seed)]
    if kind == "batch":
        out = []
        for k in range(case["n"]):
            # (the sweep's boxes are the same for every seed, their states are not)
            rng = np.random.default_rng([77, k])
            out.append(_packed(int(rng.integers(500, case["nmax"] + 1)), seed + 1000 * (k + 1),
                               kn=float(10.0 ** rng.uniform(3.0, 4.2)),
                               en=float(rng.uniform(0.3, 0.95)),
                               muc=float(rng.uniform(0.1, 0.8)),
                               radius=float(rng.uniform(0.8e-3, 1.2e-3))))
        return out
    return [scenarios.adjoint_box(n=case["n"], seed=seed)]


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())


def _dp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def prepare(case, seed):
    with tempfile.TemporaryDirectory() as d:
        if case["kind"] == "adjoint":
            return _prepare_adjoint(case, seed, Path(d))
        if case["kind"] == "pour":
            tet = scenarios.write_tetrahedron(Path(d) / "tet.insert")
            scenes = [scenarios.convex_pour(n=case["n"], seed=seed, poly_path=tet, vmax=0.5,
                                            cylinders=case["cylinders"])]
        else:
            scenes = _scenes(case, seed)
        xmls = [str(s.write_xml(Path(d) / f"s{k}.xml")) for k, s in enumerate(scenes)]
        g = Grains(xmls, FP64 if case["precision"] == "fp64" else FP32_SPLIT)
        inst, typ, x, v, w, q = scenarios.concat_state(scenes)
        g.upload_state(typ, x, v, w, q, inst=inst)
        g.do_before_time_stepping()
    if case["kind"] == "pour":
        g.step(case["warm"])            # the first bodies meet
    out = {k: _pinned((g.n, c)) for k, c in (("x", 3), ("v", 3), ("w", 3), ("q", 4), ("F", 3),
                                            ("T", 3))}
    state = dict(g=g, out=out, steps=case["steps"])
    if case["kind"] == "coupled":
        state["hydro"] = _drag(case["n"], seed)
    return state


def _drag(n, seed):
    """A fluid's forces and torques: a few percent of a sphere's weight."""
    rng = np.random.default_rng([seed, 77])
    return rng.normal(0.0, 3.0e-6, size=(n, 3)), rng.normal(0.0, 1.0e-9, size=(n, 3))


def _prepare_adjoint(case, seed, d):
    sc = scenarios.adjoint_box(n=case["n"], seed=seed)
    xml = sc.write_xml(d / "adj.xml")
    adj = Adjoint(xml)
    adj.set_particles(sc.type, sc.x, sc.v)
    tx, tv, _ = adj.run(np.array(P_TARGET), case["steps"])
    return dict(adj=adj, tx=tx, tv=tv, steps=case["steps"], every=case["every"],
                params=np.array(P_START))


def run(state):
    if "adj" in state:
        loss, gp, gv = state["adj"].gradients(state["params"], state["tx"], state["tv"],
                                              state["steps"], every=state["every"])
        return dict(loss=loss, dparams=gp, dv0=gv)
    g, o = state["g"], state["out"]
    if "hydro" in state:
        g.set_hydro_forces(*state["hydro"])
    g.step(state["steps"])
    # Grains.download_state into the program's own pinned buffers
    rc = library().gdem_download_state(g._h, _dp(o["x"]), _dp(o["v"]), _dp(o["w"]), None,
                                       _dp(o["q"]), _dp(o["F"]), _dp(o["T"]))
    if rc:
        raise RuntimeError(library().gdem_last_error().decode())
    return o


def _particles(case):
    if case["kind"] == "batch":
        return case["n"] * (500 + case["nmax"]) // 2
    return case["n"]


def work(case):
    """State in and out at every step (x, v, w, q; w in the body frame and the
    orientation matrix too where bodies are not spheres), the memory of the
    lasting contacts read and written, the state to the host once."""
    n, steps = _particles(case), case["steps"]
    if case["kind"] == "adjoint":
        # forward, recomputed forward and reverse: about 2 contacts a particle
        return {"bytes": 3 * steps * n * (2 * 120 + 2 * 2 * 48), "flops": steps * n * 2 * 2500.0}
    state = 13 * 8 + (12 * 8 if case["kind"] == "pour" else 0)
    per_step = 2 * state
    contacts = {"bed": 3.0, "coupled": 3.0, "batch": 3.0, "gas": 0.01, "pour": 0.05}[case["kind"]]
    if case.get("law", "HookeMemory") == "HookeMemory":
        per_step += contacts * 2 * (72 if case["precision"] == "fp64" else 36)
    return {"bytes": steps * n * per_step + n * 19 * 8,
            "flops": steps * n * (150.0 + 300.0 * contacts)}


def tolerance(case):
    """About four times what one changed rounding makes of the results.

    A contact whose tangential force switches branch (rest to sliding, the
    spring's cap) jumps, and every collision magnifies a difference, so the
    tails are far above the rounding of a single force.  FP64: positions
    perturbed in their last bit move the forces by up to 2e-7 (rel) and 1e-5
    (max) over two passes.  FP32-split against FP64 from the same start:
    3.6e-4 / 3e-3 in the beds, 1e-3 / 0.3 in the gas and in the sweep (whose
    boxes differ in friction and slide more), 1e-6 / 2e-5 in the pours
    (3e-4 in the torque of a cylinder that only just touches).  The gradients
    differ from those of plain autograd by 8e-9."""
    if case["kind"] == "adjoint":
        return {"rel": 4e-8, "max": 4e-6}
    if case["precision"] == "fp64":
        return {"rel": 1e-6, "max": 1e-4}
    return {"bed": {"rel": 1.5e-3, "max": 0.05}, "coupled": {"rel": 1e-4, "max": 0.01},
            "gas": {"rel": 4e-3, "max": 0.9}, "batch": {"rel": 5e-3, "max": 0.9},
            "pour": {"rel": 1e-4, "max": 2e-3}}[case["kind"]]


# ------------------------------------------------- the step in 64-bit torch --
class _Reference:
    """Second-order leapfrog of spheres with the Hooke / HookeMemory law in
    plain torch float64, every contact of a step at once."""

    def __init__(self, scenes, dev, grad=False):
        self.dev, self.grad = dev, grad
        f = lambda a: torch.as_tensor(np.asarray(a, dtype=np.float64), device=dev)
        self.x, self.v, self.w, self.q = (f(np.concatenate([getattr(s, k) for s in scenes]))
                                          for k in ("x", "v", "w", "q"))
        s0 = scenes[0]
        self.n, self.dt = len(self.x), s0.dt
        inst = np.concatenate([np.full(s.n, k) for k, s in enumerate(scenes)])
        per_type = lambda key: f(np.concatenate(
            [np.array([t[key] for t in s.types])[s.type] for s in scenes]))
        self.r = per_type("radius")
        self.mass = per_type("density") * (4.0 / 3.0) * math.pi * self.r ** 3
        self.inertia = 0.4 * self.mass * self.r ** 2
        self.weight = self.mass[:, None] * f(s0.gravity)
        self.inst = torch.as_tensor(inst, device=dev)
        self.L = f(s0.maxc) - f(s0.origin)
        self.org = f(s0.origin)
        self.per = torch.as_tensor(np.asarray(s0.periodic, bool), device=dev)
        # instances side by side for the pair search only
        self.span = max(float(np.max(s.maxc)) for s in scenes) + 0.1
        self.law = s0.models[0].get("law", "HookeMemory")
        par = lambda key, row: f([(s.models[min(row, len(s.models) - 1)].get(key) or 0.0)
                                  for s in scenes])[self.inst]
        self.par = [{k: par(k, row) for k in ("kn", "en", "muc", "kt", "mur", "kr")}
                    for row in (0, 1)]
        self.walls = []
        if s0.walls:
            for k in range(6):
                d, side = k // 2, k % 2
                face = f([(0.0 if side == 0 else s.maxc[d]) for s in scenes])[self.inst]
                req = f([(0.75 / math.pi * float(np.prod(s.walls[k]["size"]))) ** (1.0 / 3.0)
                         for s in scenes])[self.inst]
                self.walls.append((d, 1.0 if side == 0 else -1.0, face, req))
        self.skin = 0.25 * float(self.r.max())
        self.i = torch.zeros(0, dtype=torch.long, device=dev)
        self.j = self.i
        self.step_no = 0
        self._fresh()
        self.wh = [self._blank(self.n) for _ in self.walls]
        self.build()

    def _blank(self, m):
        z = lambda: torch.zeros(m, 3, dtype=torch.float64, device=self.dev)
        return dict(kd=z(), pn=z(), sp=z(),
                    last=torch.full((m,), -2, dtype=torch.long, device=self.dev))

    def _fresh(self):
        self.h = self._blank(len(self.i))

    def build(self):
        """Pairs closer than the skin, each once, with the memory carried over."""
        x = self.x.detach()
        cut = 2.0 * float(self.r.max()) + self.skin
        lo = x - self.org
        ext = self.L.clone()
        ncell = torch.clamp((ext / cut).floor(), min=1)
        edge = ext / ncell
        # (the box of another instance can be larger: cells beyond are clamped)
        c = torch.clamp((lo / edge).floor(), min=0)
        nc = [int(max(float(ncell[d]), float(c[:, d].max()) + 1)) for d in range(3)]
        c = torch.minimum(c, torch.tensor(nc, device=self.dev, dtype=c.dtype) - 1).long()
        code = lambda a: ((self.inst * nc[0] + a[:, 0]) * nc[1] + a[:, 1]) * nc[2] + a[:, 2]
        key = code(c)
        skey, order = torch.sort(key)
        ids = torch.arange(self.n, device=self.dev)
        found = []
        offs = [(a, b, e) for a in (-1, 0, 1) for b in (-1, 0, 1) for e in (-1, 0, 1)]
        seen = set()
        for o in offs:
            # in a direction of fewer than 3 periodic cells an offset repeats
            norm = tuple((o[d] % nc[d]) if self.per[d] else o[d] for d in range(3))
            if norm in seen:
                continue
            seen.add(norm)
            cc = c + torch.tensor(o, device=self.dev)
            ok = torch.ones(self.n, dtype=torch.bool, device=self.dev)
            for d in range(3):
                if self.per[d]:
                    cc[:, d] %= nc[d]
                else:
                    ok &= (cc[:, d] >= 0) & (cc[:, d] < nc[d])
            a = ids[ok]
            k = code(torch.cat([cc[ok]])) if ok.all() else \
                ((self.inst[ok] * nc[0] + cc[ok, 0]) * nc[1] + cc[ok, 1]) * nc[2] + cc[ok, 2]
            b0 = torch.searchsorted(skey, k)
            cnt = torch.searchsorted(skey, k, right=True) - b0
            a2 = torch.repeat_interleave(a, cnt)
            first = torch.repeat_interleave(b0 - (torch.cumsum(cnt, 0) - cnt), cnt)
            u = order[first + torch.arange(len(a2), device=self.dev)]
            up = a2 < u
            a2, u = a2[up], u[up]
            d2 = (self.between(x, a2, u) ** 2).sum(1)
            near = d2 < (self.r[a2] + self.r[u] + self.skin) ** 2
            found.append(a2[near] * self.n + u[near])
        new = torch.unique(torch.cat(found))
        old_i, old_j, old = self.i, self.j, self.h
        self.i, self.j = new // self.n, new % self.n
        self._fresh()
        if len(old_i) and len(new):
            live = (old["last"] == self.step_no).nonzero().flatten()
            at = torch.searchsorted(new, old_i[live] * self.n + old_j[live]).clamp(max=len(new) - 1)
            hit = new[at] == old_i[live] * self.n + old_j[live]
            live, at = live[hit], at[hit]
            self.h = {k: self.h[k].index_copy(0, at, old[k][live]) for k in self.h}
        self.x_built = x.clone()

    def between(self, x, a, b):
        d = x[b] - x[a]
        if self.per.any():
            d = torch.where(self.per, d - self.L * torch.round(d.detach() / self.L), d)
        return d

    def contact(self, p, idx, pen, lev0, lev1, v0, w0, v1, w1, mi, ri, h, at):
        """Force on body 0, its rolling torque, and the memory updated in place
        of the rows `at` of h; mi, ri: reduced mass and radius."""
        dot = lambda a, b: (a * b).sum(1, keepdim=True)
        nrm = lambda a: a.norm(dim=1, keepdim=True)
        cross = lambda a, b: torch.linalg.cross(a, b)
        g = {k: t[idx][:, None] if t.dim() else t for k, t in p.items()}
        n = pen / nrm(pen)
        n = torch.where(n.abs() < 1e-10, torch.zeros_like(n), n)
        rel = (v0 + cross(w0, lev0)) - (v1 + cross(w1, lev1))
        vn = n * dot(rel, n)
        vt = rel - vn
        beta = torch.log(g["en"]) / torch.sqrt(math.pi ** 2 + torch.log(g["en"]) ** 2)
        gn = -2.0 * beta * torch.sqrt(mi * g["kn"])
        fn = g["kn"] * pen - gn * vn
        nfn = nrm(fn)
        gt = 2.0 * (-beta * torch.sqrt(g["kn"] / mi)) * mi
        visc = -gt * vt
        zero = torch.zeros_like(fn)
        if self.law == "Hooke":
            nv = nrm(vt)
            ft = torch.where(g["muc"] * nfn < nrm(visc), -vt / nv * (g["muc"] * nfn), visc)
            wr = w0 - w1
            nw = nrm(wr)
            slip = nrm(cross(w1, lev1) - cross(w0, lev0))
            mr = torch.where(nw > 1e-10, -(g["kr"] * ri * nfn * slip / nw) * wr, zero)
            h["last"][at] = self.step_no
            return fn + ft, torch.where(nw > 1e-10, mr, zero)
        was = (h["last"][at] == self.step_no - 1)[:, None]
        pn, kd, sp = h["pn"][at], h["kd"][at], h["sp"][at]
        pn = torch.where(was, pn, n)
        # the rotation taking the previous normal to this one
        qw = torch.sqrt(dot(pn, pn) * dot(n, n)) + dot(pn, n)
        qv = cross(pn, n)
        qn = torch.sqrt(dot(qv, qv) + qw * qw)
        qv, qw = qv / qn, qw / qn
        rot = lambda a: (qw * qw - dot(qv, qv)) * a + 2.0 * dot(a, qv) * qv + 2.0 * qw * cross(qv, a)
        kd = torch.where(was, rot(kd), zero) + self.dt * g["kt"] * vt
        nut = nrm(vt)
        s = kd + gt * vt
        t = torch.where(nut > 0.001, -vt / nut, -s / nrm(s))
        nft = nrm(-kd + visc)
        stick = nft <= g["muc"] * nfn
        kd = torch.where(stick, kd, ((-g["muc"] * nfn) * t + visc) / g["kt"])
        ft = torch.where(stick, nft, g["muc"] * nfn) * t
        mr = zero
        if float(g["mur"].max()) > 0.0 if len(idx) else False:
            wr = w0 - w1
            kr = 3.0 * g["kn"] * (g["mur"] * ri) ** 2
            cap = g["mur"] * ri * nfn
            sp = torch.where(was, rot(sp), zero) - kr * self.dt * wr
            ns = nrm(sp)
            sp = torch.where(ns > cap, sp * (cap / ns), sp)
            mr = sp
        if self.grad:
            h["kd"], h["pn"] = h["kd"].index_copy(0, at, kd), h["pn"].index_copy(0, at, n)
        else:
            h["kd"][at], h["pn"][at], h["sp"][at] = kd, n, sp
        h["last"][at] = self.step_no
        return fn + ft, mr

    def forces(self, v, w):
        x = self.x
        d = x.detach() - self.x_built
        if self.per.any():
            d = torch.where(self.per, d - self.L * torch.round(d / self.L), d)
        if float((d * d).sum(1).max()) > (0.5 * self.skin) ** 2:
            self.step_no -= 1              # the memory is the previous evaluation's
            self.build()
            self.step_no += 1
        F = self.weight.clone()
        T = torch.zeros_like(F)
        cross = lambda a, b: torch.linalg.cross(a, b)
        d2 = (self.between(x.detach(), self.i, self.j) ** 2).sum(1)
        at = (d2.sqrt() - (self.r[self.i] + self.r[self.j]) < 0).nonzero().flatten()
        if len(at):
            i, j = self.i[at], self.j[at]
            ab = self.between(x, i, j)
            dist = ab.norm(dim=1, keepdim=True)
            ov = dist - (self.r[i] + self.r[j])[:, None]
            lev0 = (self.r[i][:, None] + 0.5 * ov) * ab / dist
            mi = (1.0 / (1.0 / self.mass[i] + 1.0 / self.mass[j]))[:, None]
            ri = (1.0 / (1.0 / self.r[i] + 1.0 / self.r[j]))[:, None]
            f, mr = self.contact(self.par[0], i, ov * ab / dist, lev0, lev0 - ab, v[i], w[i],
                                 v[j], w[j], mi, ri, self.h, at)
            F = F.index_add(0, i, f).index_add(0, j, -f)
            T = T.index_add(0, i, cross(lev0, f) + mr)
            T = T.index_add(0, j, -(cross(lev0 - ab, f) + mr))
        for (ax, sign, face, req), h in zip(self.walls, self.wh):
            ov = sign * (x[:, ax] - face) - self.r
            at = (ov.detach() < 0).nonzero().flatten()
            if not len(at):
                continue
            e = torch.zeros(1, 3, dtype=torch.float64, device=self.dev)
            e[0, ax] = -sign
            o = ov[at][:, None]
            lev0 = e * (self.r[at][:, None] + 0.5 * o)
            zero = torch.zeros_like(lev0)
            f, mr = self.contact(self.par[1], at, e * o, lev0, zero, v[at], w[at], zero, zero,
                                 (1.0 / (1.0 / self.mass[at] + 1.0e-20))[:, None],
                                 (1.0 / (1.0 / self.r[at] + 1.0 / req[at]))[:, None], h, at)
            F = F.index_add(0, at, f)
            T = T.index_add(0, at, cross(lev0, f) + mr)
        return F, T

    def start(self):
        self.F, self.T = self.forces(self.v, self.w)
        for h in [self.h, *self.wh]:
            h["kd"] = torch.zeros_like(h["kd"])
            h["sp"] = torch.zeros_like(h["sp"])

    def advance(self, steps, hydro=None):
        hm, hi = 0.5 * self.dt / self.mass[:, None], 0.5 * self.dt / self.inertia[:, None]
        for _ in range(steps):
            # (the fluid's forces join at every kick; F and T are the contacts' and the weight)
            fx, tx = (0.0, 0.0) if hydro is None else hydro
            v, w = self.v + (self.F + fx) * hm, self.w + (self.T + tx) * hi
            x = self.x + v * self.dt
            if self.per.any():
                x = torch.where(self.per, x - self.L * torch.floor((x.detach() - self.org) / self.L),
                                x)
            self.x = x
            if not self.grad:
                om = w.norm(dim=1, keepdim=True)
                half = om * (0.5 * self.dt)
                a = torch.where(om > 1e-10, torch.sin(half) / om.clamp(min=1e-300) * w,
                                torch.zeros_like(w))
                aw = torch.where(om > 1e-10, torch.cos(half), torch.ones_like(half))
                qv, qw = self.q[:, :3], self.q[:, 3:]
                self.q = torch.cat([torch.linalg.cross(a, qv) + aw * qv + qw * a,
                                    aw * qw - (a * qv).sum(1, keepdim=True)], dim=1)
            self.step_no += 1
            self.F, self.T = self.forces(v, w)
            self.v, self.w = v + (self.F + fx) * hm, w + (self.T + tx) * hi


def exact(case, seed):
    """run()'s first answer in 64 bits (None for bodies that are not spheres:
    their closest-point search has no plain form)."""
    if case["kind"] == "pour":
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    scenes = _scenes(case, seed)
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, scenes, dev)
    with torch.no_grad():
        ref = _Reference(scenes, dev)
        ref.start()
        hydro = None
        if case["kind"] == "coupled":
            hydro = [torch.as_tensor(a, device=dev) for a in _drag(case["n"], seed)]
        ref.advance(case["steps"], hydro)
    return dict(x=ref.x, v=ref.v, w=ref.w, q=ref.q, F=ref.F, T=ref.T)


def _exact_adjoint(case, scenes, dev):
    def setup(params, grad):
        ref = _Reference(scenes, dev, grad)
        for p in ref.par:
            for k, t in zip(("kn", "en", "muc"), params):
                p[k] = t.expand(ref.n) if t.dim() == 0 else t
        return ref

    f = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
    with torch.no_grad():
        target = setup([f(a) for a in P_TARGET], False)
        target.start()
        target.advance(case["steps"])
    params = [f(a).requires_grad_() for a in P_START]
    ref = setup(params, True)
    v0 = ref.v.clone().requires_grad_()
    ref.v = v0
    ref.start()
    ref.advance(case["steps"])
    loss = ((ref.x - target.x) ** 2).sum() + ((ref.v - target.v) ** 2).sum()
    gp = torch.autograd.grad(loss, [*params, v0])
    return dict(loss=float(loss.detach()), dparams=torch.stack(gp[:3]), dv0=gp[3])
