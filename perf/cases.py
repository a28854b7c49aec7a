"""The calls whose time counts, as a program that uses this library makes them.

A program keeps a solver (or the batched server) and host buffers, and per pass
advances the flow by one output interval and reads the result back; two kinds
hand whole solves over.  The kinds, each over the range of its `draw`:

  vortex    one component, periodic (Taylor-Green vortex and seeded modes)
  droplets  two components with density ratio in a periodic box, with the phi
            mass correction or the film repulsion where a run asks for them
  channel   two components between walls, around solid spheres, with wetting
  porous    one component driven by pressure faces through solid spheres with
            half-way bounce-back
  handover  a state continued from host data: uploaded, advanced, downloaded
  server    a mix of small solves through the batched server

`exact` restates the scheme in plain torch, in 64 bits.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import lbfast_b200 as lbf
from lbfast_b200.capi import check

# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # the Taylor-Green check of the reference: a small box, where launches and latency count
        dict(name="taylor_green_64", kind="vortex", lx=64, ly=64, lz=64, lattice=19, highorder=0, smag=0, storage="f32",
             steps=100),
        # the smallest two-component box that is served, a few steps at a time (a probe in a parameter scan)
        dict(name="droplet_32", kind="droplets", lx=32, ly=32, lz=32, lattice=27, highorder=1, storage="f32", steps=10,
             drops=1, ratio=10.0, option="none"),
        # the Laplace droplet box of the benchmark, its density ratio of 100
        dict(name="laplace_256", kind="droplets", lx=256, ly=256, lz=256, lattice=27, highorder=1, storage="f32",
             steps=40, drops=1, ratio=100.0, option="none"),
        # many droplets in a large ragged box, 16-bit storage
        dict(name="emulsion_f16", kind="droplets", lx=330, ly=290, lz=250, lattice=27, highorder=1, storage="f16",
             steps=30, drops=40, ratio=10.0, option="none"),
        # the two-component channel with spheres of the benchmark
        dict(name="channel_512", kind="channel", lx=512, ly=256, lz=256, lattice=27, highorder=1, storage="f32",
             steps=20, spheres=64, drops=32, angle=90.0),
        # a turbulent one-component box with the Smagorinsky relaxation time
        dict(name="turbulence_200", kind="vortex", lx=200, ly=184, lz=168, lattice=27, highorder=1, smag=1,
             storage="f32", steps=40),
        # pressure-driven flow through a bed of spheres
        dict(name="porous_160", kind="porous", lx=160, ly=96, lz=80, lattice=19, highorder=0, storage="f32", steps=50,
             spheres=24),
        # droplets held apart by the film repulsion
        dict(name="film_112", kind="droplets", lx=112, ly=96, lz=88, lattice=27, highorder=1, storage="f32", steps=20,
             drops=12, ratio=2.0, option="repulsive"),
        # a long emulsion run that keeps its phase volume
        dict(name="emulsion_corr", kind="droplets", lx=150, ly=128, lz=136, lattice=27, highorder=1, storage="f32",
             steps=40, drops=12, ratio=10.0, option="correction"),
        # the double-precision run that others are checked against
        dict(name="droplets_f64", kind="droplets", lx=96, ly=88, lz=104, lattice=27, highorder=1, storage="f64",
             steps=20, drops=4, ratio=10.0, option="none"),
        # a state from another program, continued for a few steps and handed back
        dict(name="handover_128", kind="handover", lx=128, ly=120, lz=136, lattice=27, highorder=1, storage="f16",
             steps=8, drops=6, ratio=10.0),
        # served droplet solves of uneven boxes
        dict(name="server_mix", kind="server", edges="32,40,48,64,32,36,56,64,32,48,33,60", storage="f16", steps=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vortex", "droplets", "droplets", "channel", "porous", "handover", "server"])
    edge = _log(rng, 28, 250)
    box = dict(lx=max(20, int(edge * rng.uniform(0.8, 1.6))), ly=max(20, int(edge * rng.uniform(0.7, 1.2))),
               lz=max(20, int(edge * rng.uniform(0.7, 1.2))))
    n = box["lx"] * box["ly"] * box["lz"]
    steps = max(4, min(100, int(4.0e8 / n), _log(rng, 10, 100)))
    storage = rng.choice(["f32", "f32", "f16", "bf16"] + (["f64"] if n < 3_000_000 else []))
    lattice, highorder = rng.choice([(15, 0), (19, 0), (27, 0), (27, 1), (27, 1)])
    drops = rng.randint(1, 12)
    if kind == "vortex":
        return dict(box, kind=kind, lattice=lattice, highorder=highorder, smag=rng.randint(0, 1), storage=storage,
                    steps=steps)
    if kind == "droplets":
        option = rng.choice(["none", "none", "correction"] + (["repulsive"] if n < 4_000_000 and storage != "f64" else []))
        return dict(box, kind=kind, lattice=lattice, highorder=highorder, storage=storage, steps=steps, drops=drops,
                    ratio=rng.choice([1.0, 2.0, 10.0]), option=option)
    if kind == "channel":
        return dict(box, kind=kind, lattice=27, highorder=rng.randint(0, 1), storage=storage, steps=steps,
                    spheres=rng.randint(0, 12), drops=drops, angle=rng.choice([60.0, 90.0, 120.0]))
    if kind == "porous":
        return dict(box, kind=kind, lattice=rng.choice([19, 27]), highorder=0,
                    storage=rng.choice(["f32", "f64"] if n < 3_000_000 else ["f32"]), steps=steps,
                    spheres=rng.randint(1, 16))
    if kind == "handover":
        return dict(box, kind=kind, lattice=lattice, highorder=highorder, storage=storage, steps=rng.randint(2, 10),
                    drops=drops, ratio=rng.choice([1.0, 10.0]))
    edges = ",".join(str(rng.randint(24, 72)) for _ in range(rng.randint(4, 14)))
    return dict(kind="server", edges=edges, storage=rng.choice(["f32", "f16"]), steps=rng.choice([40, 64, 96]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _grid(c):
    ax = [torch.arange(n, device=_dev(), dtype=torch.float64) for n in (c["lz"], c["ly"], c["lx"])]
    return ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]


def _modes(c, rng, amp):
    """A smooth solenoidal-like velocity: a Taylor-Green vortex and a few seeded modes, amplitude amp."""
    z, y, x = _grid(c)
    kx, ky, kz = (2 * math.pi / n for n in (c["lx"], c["ly"], c["lz"]))
    u = torch.sin(kx * x) * torch.cos(ky * y) * torch.cos(kz * z)
    v = -torch.cos(kx * x) * torch.sin(ky * y) * torch.cos(kz * z)
    w = torch.zeros_like(u)
    for _ in range(3):
        a, b, d = rng.uniform(0.1, 0.4, 3)
        p, q, r = rng.uniform(0, 2 * math.pi, 3)
        m = int(rng.integers(1, 4))
        u = u + a * torch.sin(m * ky * y + p)
        v = v + b * torch.sin(m * kz * z + q)
        w = w + d * torch.sin(m * kx * x + r)
    return amp * u, amp * v, amp * w


def _periodic(d, n):
    return d - n * torch.round(d / n)


def _phi(c, rng, n, width):
    """n seeded droplets with the tanh profile; phi in [0, 1] and the Laplace pressure factor 2 phi / R."""
    z, y, x = _grid(c)
    lo = min(c["lx"], c["ly"], c["lz"])
    phi = torch.zeros(c["lz"], c["ly"], c["lx"], device=_dev(), dtype=torch.float64)
    curv = torch.zeros_like(phi)
    for _ in range(n):
        r = rng.uniform(0.14, 0.24) * lo if n < 16 else rng.uniform(0.06, 0.12) * lo
        cx, cy, cz = rng.uniform(0, 1, 3) * np.array([c["lx"], c["ly"], c["lz"]])
        d = torch.sqrt(_periodic(x - cx, c["lx"]) ** 2 + _periodic(y - cy, c["ly"]) ** 2 + _periodic(z - cz, c["lz"]) ** 2)
        f = 0.5 * (1.0 - torch.tanh((d - r) / (0.5 * width)))
        curv = torch.where(f > phi, 2.0 * f / r, curv)
        phi = torch.maximum(phi, f)
    return phi, curv


def _spheres(c, rng, n):
    z, y, x = _grid(c)
    lo = min(c["lx"], c["ly"], c["lz"])
    solid = torch.zeros(c["lz"], c["ly"], c["lx"], device=_dev(), dtype=torch.bool)
    for _ in range(n):
        r = rng.uniform(0.03, 0.055) * lo if n > 32 else rng.uniform(0.06, 0.11) * lo
        cx, cy, cz = (rng.uniform(r + 2.5, m - 3.5 - r) for m in (c["lx"], c["ly"], c["lz"]))
        solid |= (x - cx) ** 2 + (y - cy) ** 2 + (z - cz) ** 2 <= r * r
    return solid


def _mark(solid, pbc, lattice):
    """isfluid: 0 solid (and the walls of the non-periodic faces), -1 fluid next to solid, 1 fluid."""
    s = solid.clone()
    for axis, periodic in zip((2, 1, 0), pbc):
        if not periodic:
            s.select(axis, 0).fill_(True)
            s.select(axis, s.shape[axis] - 1).fill_(True)
    near = torch.zeros_like(s)
    for cx, cy, cz in _links(lattice)[1:]:
        near |= _at(s, (cx, cy, cz), pbc, False)
    return torch.where(s, 0, torch.where(near, -1, 1)).to(torch.int8)


def _seed_phi(phi, isf, pbc):
    """phi of the solid nodes next to fluid: the mean of their fluid neighbours; 0 deeper inside."""
    fluid = (isf != 0).to(torch.float64)
    num, den = torch.zeros_like(phi), torch.zeros_like(phi)
    for e in _links(27)[1:]:
        wgt = 1.0 / math.sqrt(sum(k * k for k in e))
        f = _at(fluid, e, pbc, 0.0)
        num += wgt * f * _at(phi, e, pbc, 0.0)
        den += wgt * f
    return torch.where(isf == 0, torch.where(den > 0, num / den.clamp_min(1e-30), torch.zeros_like(phi)), phi)


def _params(c):
    """The run parameters of a case as keywords of lbf.Params."""
    p = dict(lx=c["lx"], ly=c["ly"], lz=c["lz"], lattice=c["lattice"], highorder=c["highorder"], storage=c["storage"])
    kind = c["kind"]
    if kind == "vortex":
        return dict(p, visc1=0.01, smagorinsky=c["smag"], fx=1e-7)
    if kind == "porous":
        return dict(p, pbc_x=0, pbc_y=0, obstacles=1, bounce_back=1, visc1=0.1, openbc=1,
                    openbc_type=((1, 1), (0, 0), (0, 0)), openbc_press=((0.002, -0.002), (0.0, 0.0), (0.0, 0.0)))
    if kind == "channel":
        return dict(p, pbc_y=0, twocomponent=1, densratio=1, obstacles=1, visc1=0.05, visc2=0.2, rho_r=0.5, rho_b=1.5,
                    sigma=0.005, width=4.0, tau_diff=0.1, fx=1e-6, wettab_r=c["angle"], printphi=1)
    p = dict(p, twocomponent=1, densratio=1 if c["ratio"] > 1 else 0, visc1=0.1, visc2=0.1, rho_r=c["ratio"], rho_b=1.0,
             sigma=0.01, width=4.0, tau_diff=0.1, fx=1e-7, printphi=1)
    if c.get("option") == "correction":
        p["phi_correction"] = 1
    if c.get("option") == "repulsive":
        p.update(repulsive_flux=1, a_rep=0.05, cos_opp_t=-0.5, q_th=0.05)
    return p


def _inputs(c, seed):
    """(parameters, isfluid or None, moments (10, lz, ly, lx), phi or None), 64-bit on the device."""
    rng = np.random.default_rng(seed)
    p = _params(c)
    kind = c["kind"]
    isf = phi = None
    press = torch.zeros(c["lz"], c["ly"], c["lx"], device=_dev(), dtype=torch.float64)
    amp = {"vortex": 0.04, "channel": 0.01, "porous": 0.01}.get(kind, 0.02)
    u, v, w = _modes(c, rng, amp)
    # a mean flow: the momentum sums are then no rounding noise around zero
    u, v, w = u + 0.6 * amp, v - 0.2 * amp, w + 0.3 * amp
    if kind in ("channel", "porous"):
        pbc = (p.get("pbc_x", 1), p.get("pbc_y", 1), p.get("pbc_z", 1))
        isf = _mark(_spheres(c, rng, c["spheres"]), pbc, c["lattice"])
    if kind not in ("vortex", "porous"):
        phi, curv = _phi(c, rng, c["drops"], p["width"])
        rho = p["rho_r"] * phi + (1 - phi) * p["rho_b"] if p["densratio"] else torch.ones_like(phi)
        press = press + 3.0 * p["sigma"] * curv / rho
    else:
        press = press + 0.005 + 0.002 * torch.cos(2 * math.pi / c["lx"] * _grid(c)[2] + rng.uniform(0, 6))
    if isf is not None:
        fluid = (isf != 0).to(torch.float64)
        u, v, w, press = u * fluid, v * fluid, w * fluid, press * fluid
        if phi is not None:
            phi = _seed_phi(phi * fluid, isf, pbc)
    mom = torch.stack([press, u, v, w, u * u, v * v, w * w, u * v, u * w, v * w])
    del press, u, v, w
    # what a program hands over: 32-bit fields (64-bit for a double-precision run)
    if c["storage"] != "f64":
        mom = mom.float()
        phi = None if phi is None else phi.float()
    return p, isf, mom, phi


def _host(t):
    """A page-locked host copy, as a program that exchanges fields often keeps them."""
    if t is None:
        return None
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=torch.cuda.is_available())
    h.copy_(t)
    return h


def _solves(c, seed):
    """The solves of a server case: one droplet box each."""
    out = []
    for i, e in enumerate(int(x) for x in c["edges"].split(",")):
        one = dict(kind="solve", lx=e, ly=e, lz=e, lattice=27, highorder=1, storage=c["storage"], drops=1,
                   ratio=10.0)
        out.append((one, seed * 1009 + i))
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "server":
        jobs = []
        for one, sd in _solves(c, seed):
            p, _, mom, phi = _inputs(one, sd)
            jobs.append((lbf.Params(**p), mom.cpu().numpy(), phi.cpu().numpy()))
        return dict(case=c, server=lbf.Server(chunk=32), jobs=jobs)
    p, isf, mom, phi = _inputs(c, seed)
    s = lbf.Solver(lbf.Params(**p))
    if isf is not None:
        s.set_isfluid(isf.cpu().numpy())
    st = dict(case=c, solver=s)
    shape = (c["lz"], c["ly"], c["lx"])
    pin = torch.cuda.is_available()
    if c["kind"] == "handover":
        st["dtype"] = 1 if c["storage"] == "f64" else 0
        st["mom"], st["phi"] = _host(mom), _host(phi)
        for key, t in (("mom_out", (10,) + shape), ("phi_out", shape), ("u_out", (3,) + shape)):
            st[key] = torch.empty(t, dtype=mom.dtype, pin_memory=pin)
    else:
        s.set_fields(mom.cpu().numpy(), None if phi is None else phi.cpu().numpy())
        for key, t in (("rho", shape), ("vel", shape + (3,)), ("press", shape)):
            st[key] = torch.empty(t, dtype=torch.float32, pin_memory=pin)
    return st


def _vp(t):
    return None if t is None else C.c_void_p(t.data_ptr())


def _fp(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def run(state):
    c = state["case"]
    if c["kind"] == "server":
        srv = state["server"]
        ids = [srv.submit(p, mom, phi, nsteps=c["steps"]) for p, mom, phi in state["jobs"]]
        srv.drain()
        return [srv.fetch(i) for i in ids]
    s = state["solver"]
    if c["kind"] == "handover":
        check(s.lib.lbf_set_fields(s.h, _vp(state["mom"]), _vp(state["phi"]), state["dtype"]))
        s.step(c["steps"])
        mom, phi, u = state["mom_out"], state["phi_out"], state["u_out"]
        check(s.lib.lbf_get_fields(s.h, _vp(mom), _vp(phi), _vp(u), state["dtype"]))
        return {"press": mom[0], "vel": mom[1:4], "pi": mom[4:], "phi": phi, "uold": u}
    # half an interval, the run's sums (a program watches them to stop a run
    # that blew up), the other half, and the printed fields
    s.step(c["steps"] // 2)
    sums = s.reduce()
    s.step(c["steps"] - c["steps"] // 2)
    check(s.lib.lbf_get_print_fields(s.h, _fp(state["rho"]), _fp(state["vel"]), _fp(state["press"])))
    return {"sums": sums, "rho": state["rho"], "vel": state["vel"], "press": state["press"]}


def work(case):
    c = case
    if c["kind"] == "server":
        n = sum(int(e) ** 3 for e in c["edges"].split(","))
    else:
        n = c["lx"] * c["ly"] * c["lz"]
    one = c["kind"] in ("vortex", "porous")
    wide = {"f32": 4, "f64": 8}.get(c["storage"])
    # per node and step, read and written: ten moments, and with two components
    # the previous velocity and phi; 16-bit storage keeps P, u, v, w and phi in 32 bits
    if wide:
        per = 2 * wide * (10 if one else 14)
    else:
        per = 2 * (4 * 4 + 6 * 2) if one else 2 * (4 * 4 + 9 * 2 + 4)
    if c["kind"] in ("channel", "porous"):
        per += 1  # isfluid
    host = 8 if c["storage"] == "f64" else 4
    if c["kind"] in ("handover", "server"):
        io = n * host * (11 + 14)
    else:
        io = n * 4 * 5
    # arithmetic of a node's collision, streaming sums and phase-field stencils
    flops = {15: 200, 19: 250, 27: 350}[c.get("lattice", 27)] + (150 if c.get("highorder", 1) else 0) + (0 if one else 450)
    return {"bytes": float(n * per * c["steps"] + io), "flops": float(n * flops * c["steps"])}


def tolerance(case):
    c = case
    # measured against `exact`, times about four (32-bit: up to 2.6e-5, of the
    # pressure; 16-bit: 2.1e-4 of the velocity with 11 significant bits, 1.6e-3
    # with 8).  A pass is tens of steps, each of which rounds its state; "max"
    # is wide where a node's neighbour is chosen by a comparison
    if c["storage"] == "f64":
        return {"rel": 1e-6, "max": 1e-4}  # the printed fields are 32-bit
    if c["storage"] == "bf16":
        return {"rel": 1e-2, "max": 0.9}
    if c["storage"] == "f16":
        return {"rel": 2e-3, "max": 0.5}
    return {"rel": 1e-4, "max": 0.3 if c.get("option") == "repulsive" else 0.02}


# ---------------------------------------------------------------------------
# the scheme in 64 bits
# ---------------------------------------------------------------------------


def _links(lattice):
    """The link vectors of D3Q27 in rising length; D3Q19 without the cube's corners, D3Q15 without its edges."""
    every = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]
    every.sort(key=lambda e: sum(k * k for k in e))
    keep = {27: (0, 1, 2, 3), 19: (0, 1, 2), 15: (0, 1, 3)}[lattice]
    return [e for e in every if sum(k * k for k in e) in keep]


# the reference's own order of the links, which decides ties between wetting donors
_ORDER = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (0, 1, 1), (0, 1, -1), (1, 0, 1), (-1, 0, 1),
          (1, 1, 1), (1, -1, 1), (-1, -1, 1), (1, -1, -1)]
_ORDER = [tuple(s * k for k in e) for e in _ORDER for s in (1, -1)]

_WEIGHT = {27: (8 / 27, 2 / 27, 1 / 54, 1 / 216), 19: (1 / 3, 1 / 18, 1 / 36, 0.0), 15: (2 / 9, 1 / 9, 0.0, 1 / 72)}


def _at(f, e, pbc, fill):
    """f at x + e; `fill` beyond a non-periodic face."""
    g = f
    for axis, k, periodic in zip((2, 1, 0), e, pbc):
        if k:
            g = torch.roll(g, -k, dims=axis - 3)
            if not periodic:
                n = g.shape[axis - 3]
                g.select(axis - 3, n - 1 if k > 0 else 0).fill_(fill)
    return g


class _Exact:
    def __init__(self, p, isf, mom, phi):
        self.p = dict(dict(pbc_x=1, pbc_y=1, pbc_z=1, twocomponent=0, densratio=0, obstacles=0, visc1=0.1, visc2=0.1,
                           rho_r=1.0, rho_b=1.0, sigma=0.0, width=4.0, tau_diff=0.1, fx=0.0, fy=0.0, fz=0.0,
                           wettab_r=90.0, phi_correction=0, smagorinsky=0, openbc=0, bounce_back=0, repulsive_flux=0,
                           highorder=0), **p)
        q = self.p
        self.pbc = (q["pbc_x"], q["pbc_y"], q["pbc_z"])
        self.tc, self.dr = bool(q["twocomponent"]), bool(q["densratio"])
        self.isf = isf
        self.fluid = None if isf is None else isf != 0
        self.mom = mom.double()
        self.uold = self.mom[1:4].clone()
        self.links = _links(q["lattice"])
        self.n = 0
        if self.tc:
            self.phi = phi.double()
            self.other = self.phi.clone()  # the second time level's phi: its solid nodes have a history of their own
            self.pending = None
            self.beta, self.kappa = 12.0 * q["sigma"] / q["width"], 1.5 * q["sigma"] * q["width"]
            self.sharp = 4.0 * q["tau_diff"] / q["width"]
            self.sum0 = self._sum(self.phi)
            if isf is not None:
                self._wet_tables()
                self.phi = self._wet(self.phi, None)

    def _sum(self, f):
        return f.sum() if self.fluid is None else f[self.fluid].sum()

    # ---- stencils ----
    def _grad(self, f, fill=0.0):
        g = [torch.zeros_like(f) for _ in range(3)]
        for e in _links(27)[1:]:
            wgt = 3.0 * _WEIGHT[27][sum(k * k for k in e)]
            h = _at(f, e, self.pbc, fill)
            for d in range(3):
                if e[d]:
                    g[d] += (wgt * e[d]) * h
        return g

    def _lap(self, f):
        s = (_WEIGHT[27][0] - 1.0) * f
        for e in _links(27)[1:]:
            s = s + _WEIGHT[27][sum(k * k for k in e)] * _at(f, e, self.pbc, 0.0)
        return 6.0 * s

    # ---- wetting ghost values ----
    def _wet_tables(self):
        lz, ly, lx = self.isf.shape
        f = self.isf.to(torch.int8)
        wn = [torch.zeros(f.shape, device=f.device, dtype=torch.float64) for _ in range(3)]
        near = {}
        for e in _ORDER:
            near[e] = _at(f, e, self.pbc, 1) != 0
            sc = 1.0 / sum(k * k for k in e)
            for d in range(3):
                if e[d]:
                    wn[d] -= sc * e[d] * near[e]
        mag = torch.sqrt(wn[0] ** 2 + wn[1] ** 2 + wn[2] ** 2)
        k, j, i = torch.nonzero((f == 0) & (mag >= 1e-14), as_tuple=True)
        wn = [c[k, j, i] / mag[k, j, i] for c in wn]
        best = torch.full(k.shape, -1e30, device=f.device, dtype=torch.float64)
        shift = torch.zeros((3,) + k.shape, device=f.device, dtype=torch.long)
        for e in _ORDER:
            # the reference's own expression: rounding decides between equal donors
            score = (-e[0] * wn[0] + -e[1] * wn[1] + -e[2] * wn[2]) * math.sqrt(1.0 / sum(c * c for c in e))
            take = near[e][k, j, i] & (score > best)
            best = torch.where(take, score, best)
            for d in range(3):
                shift[d] = torch.where(take, e[d], shift[d])
        don = [i + shift[0], j + shift[1], k + shift[2]]
        keep = (best > -1e29) & (don[0] >= 0) & (don[1] >= 0) & (don[2] >= 0)
        high = torch.zeros_like(keep)
        out = torch.zeros_like(keep)
        for d, (n, periodic) in enumerate(zip((lx, ly, lz), self.pbc)):
            over = don[d] >= n
            if periodic:
                high |= over
            else:
                out |= over
            don[d] = torch.where(over, don[d] - n, don[d])
        self.wk, self.wj, self.wi = k[keep], j[keep], i[keep]
        self.don = [torch.where(out, torch.zeros_like(c), c)[keep] for c in don]
        self.wn = [c[keep] for c in wn]
        self.shift = [-s[keep].double() for s in shift]
        self.high, self.out = high[keep], out[keep]
        t = (180.0 - self.p["wettab_r"]) * math.pi / 180.0
        self.cot = math.cos(t) / math.sin(t)

    def _ghost(self, phi, g):
        at = (self.don[2], self.don[1], self.don[0])
        old = phi[self.wk, self.wj, self.wi]
        val = phi[at]
        zero = self.out if g is not None else self.out | self.high
        if g is not None:
            gx, gy, gz = (c[at] for c in g)
            dot = gx * self.wn[0] + gy * self.wn[1] + gz * self.wn[2]
            t = [c - dot * n for c, n in zip((gx, gy, gz), self.wn)]
            mag = torch.sqrt(t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
            b = [c - mag * self.cot * n for c, n in zip(t, self.wn)]
            val = val + (b[0] * self.shift[0] + b[1] * self.shift[1] + b[2] * self.shift[2]) * (4.0 * old * (1.0 - old))
        return torch.where(zero, torch.zeros_like(val), val).clamp(0.0, 1.0)

    def _wet(self, phi, g):
        phi = phi.clone()
        phi[self.wk, self.wj, self.wi] = self._ghost(phi, g)
        return phi

    # ---- film repulsion ----
    def _repulsion(self, phi, raw):
        p, eps = self.p, 1e-9
        g = self._grad(raw)
        den = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2) + eps
        n = [c / den for c in g]
        q = phi.clamp(0.0, 1.0)
        q = q * (1.0 - q)
        r2 = torch.full_like(phi, 1e300)
        face = torch.full_like(phi, -1.0)
        off = [torch.zeros_like(phi) for _ in range(3)]
        for di in range(-3, 4):
            for dj in range(-3, 4):
                for dk in range(-3, 4):
                    if not (di or dj or dk):
                        continue
                    roll = lambda f: torch.roll(f, (-dk, -dj, -di), dims=(0, 1, 2))  # noqa: E731
                    qn = roll(q)
                    dot = n[0] * roll(n[0]) + n[1] * roll(n[1]) + n[2] * roll(n[2])
                    fac = 0.5 * (1.0 - dot)
                    d2 = float(di * di + dj * dj + dk * dk)
                    ok = (qn >= p["q_th"]) & ((qn - q).abs() <= 0.1 * q.clamp_min(1e-12)) & (dot <= p["cos_opp_t"])
                    take = ok & ((d2 < r2 - 1e-14) | (((d2 - r2).abs() <= 1e-14) & (fac > face)))
                    r2 = torch.where(take, torch.full_like(r2, d2), r2)
                    face = torch.where(take, fac, face)
                    for c, d in zip(off, (di, dj, dk)):
                        c[take] = d
        f = [torch.zeros_like(phi) for _ in range(3)]
        k, j, i = torch.nonzero((r2 < 1e299) & (q >= p["q_th"]) & (phi * (1.0 - phi) > eps), as_tuple=True)
        at = (k, j, i)
        d = [c[at] for c in off]
        to = ((k + d[2].long()) % phi.shape[0], (j + d[1].long()) % phi.shape[1], (i + d[0].long()) % phi.shape[2])
        a, b = [c[at] for c in n], [c[to] for c in n]
        r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
        d = [c / r for c in d]
        fac = (-(a[0] * b[0] + a[1] * b[1] + a[2] * b[2])).clamp_min(0.0)
        ns = [x - y for x, y in zip(a, b)]
        m = torch.sqrt(ns[0] ** 2 + ns[1] ** 2 + ns[2] ** 2)
        ns = [torch.where(m <= eps, y, x / m.clamp_min(eps)) for x, y in zip(ns, d)]
        s = torch.where(d[0] * ns[0] + d[1] * ns[1] + d[2] * ns[2] < 0, -1.0, 1.0)
        loc, far = phi[at], phi[to]
        qc = (0.5 * (loc * (1.0 - loc) + far * (1.0 - far))).clamp(eps, 0.25 - eps)
        arg = 1.0 / (2.0 * torch.sqrt(qc))
        film = p["width"] * torch.log(arg + torch.sqrt(arg * arg - 1.0))
        amp = p["a_rep"] / (1.0 + film ** 4) * qc * fac
        amp = torch.where((fac > eps) & (film > 0), amp, torch.zeros_like(amp))
        cap = 1.5 * sum((amp * x).abs() for x in ns)
        sc = (loc / cap.clamp_min(1e-9)).clamp_max(1.0)
        for c, x in zip(f, ns):
            c[at] = amp * s * x * sc
        return f

    # ---- post-collision populations, by link ----
    def _populations(self, P, vel, pi, F, om):
        u, v, w = vel
        Fx, Fy, Fz = F
        X, Y, Z, XY, XZ, YZ = (a - b for a, b in zip(pi, (u * u, v * v, w * w, u * v, u * w, v * w)))
        o = 1.0 - om
        mx, my, mz = u + 0.5 * Fx, v + 0.5 * Fy, w + 0.5 * Fz
        mxx, myy, mzz = u * u + o * X + u * Fx, v * v + o * Y + v * Fy, w * w + o * Z + w * Fz
        mxy = u * v + o * XY + 0.5 * (u * Fy + v * Fx)
        mxz = u * w + o * XZ + 0.5 * (u * Fz + w * Fx)
        myz = v * w + o * YZ + 0.5 * (v * Fz + w * Fy)
        lat = self.p["lattice"]
        if not self.p["highorder"] and lat != 27:
            base = P - 1.5 * (mxx + myy + mzz)
            for x, y, z in self.links:
                s = base + 3.0 * (x * mx + y * my + z * mz) + 4.5 * (x * x * mxx + y * y * myy + z * z * mzz)
                s = s + 9.0 * (x * y * mxy + x * z * mxz + y * z * myz)
                yield (x, y, z), _WEIGHT[lat][x * x + y * y + z * z] * s
            return
        M = {(0, 0, 0): P, (1, 0, 0): mx, (0, 1, 0): my, (0, 0, 1): mz, (2, 0, 0): mxx, (0, 2, 0): myy, (0, 0, 2): mzz,
             (1, 1, 0): mxy, (1, 0, 1): mxz, (0, 1, 1): myz}
        if self.p["highorder"]:
            u2, v2, w2 = u * u, v * v, w * w
            M[2, 1, 0] = u2 * v + o * (2 * XY * u + X * v)
            M[2, 0, 1] = u2 * w + o * (2 * XZ * u + X * w)
            M[1, 2, 0] = u * v2 + o * (Y * u + 2 * XY * v)
            M[1, 0, 2] = u * w2 + o * (Z * u + 2 * XZ * w)
            M[0, 1, 2] = v * w2 + o * (Z * v + 2 * YZ * w)
            M[0, 2, 1] = v2 * w + o * (2 * YZ * v + Y * w)
            M[1, 1, 1] = u * v * w + o * (YZ * u + XZ * v + XY * w)
            M[2, 2, 0] = u2 * v2 + o * (Y * u2 + 2 * v * (3 * XY * u + X * v))
            M[2, 0, 2] = u2 * w2 + o * (Z * u2 + 2 * w * (3 * XZ * u + X * w))
            M[0, 2, 2] = v2 * w2 + o * (Z * v2 + 2 * w * (3 * YZ * v + Y * w))
            M[1, 1, 2] = u * v * w2 + o * (Z * u * v + w * (3 * YZ * u + 3 * XZ * v + 2 * XY * w))
            M[1, 2, 1] = u * v2 * w + o * (2 * YZ * u * v + XZ * v2 + 2 * Y * u * w + 4 * XY * v * w)
            M[2, 1, 1] = u2 * v * w + o * (YZ * u2 + 2 * XZ * u * v + 4 * XY * u * w + 2 * X * v * w)
            M[2, 1, 2] = u2 * v * w2 + o * (Z * u2 * v + 3 * w * (YZ * u2 + 2 * XZ * u * v + 2 * XY * u * w + X * v * w))
            M[2, 2, 1] = u2 * v2 * w + o * (2 * u * v * (YZ * u + XZ * v) + 2 * Y * u2 * w + v * (10 * XY * u + 3 * X * v) * w)
            M[1, 2, 2] = u * v2 * w2 + o * (Z * u * v2 + 3 * w * (2 * YZ * u * v + XZ * v2 + Y * u * w + 2 * XY * v * w))
            M[2, 2, 2] = u2 * v2 * w2 + o * (Z * u2 * v2 + w * (6 * u * v * (YZ * u + XZ * v) + 3 * Y * u2 * w
                                                                + 2 * v * (7 * XY * u + 2 * X * v) * w))
        # the expansion is a product of three one-axis transforms
        T = {-1: (1 / 6, -0.5, 0.5), 0: (2 / 3, 0.0, -1.0), 1: (1 / 6, 0.5, 0.5)}

        def along(src, axis):
            out = {}
            for key, f in src.items():
                for c in (-1, 0, 1):
                    t = T[c][key[axis]]
                    if t:
                        to = key[:axis] + ("c%d" % c,) + key[axis + 1:]
                        out[to] = out[to].add_(f, alpha=t) if to in out else f * t
            return out

        M = along(along(along(M, 0), 1), 2)
        for key in list(M):
            yield tuple(int(k[1:]) for k in key), M.pop(key)

    def step(self):
        p, dr, tc = self.p, self.dr, self.tc
        P, u, v, w = self.mom[0:4]
        pi = list(self.mom[4:10])
        phi = raw = inv = None
        corr = None
        one = torch.ones_like(P)
        f = [one * p["fx"], one * p["fy"], one * p["fz"]]
        rho = one
        if tc:
            raw = self.phi
            g = self._grad(raw)
            mag = torch.sqrt(g[0] ** 2 + g[1] ** 2 + g[2] ** 2)
            n = [c / (mag + 1e-9) for c in g]
            if self.fluid is not None:
                n = [torch.where(self.fluid, c, torch.zeros_like(c)) for c in n]
                ghost = self._ghost(raw, [c * mag for c in n])
            gf = [c * mag for c in n]
            # nodes beyond a non-periodic face carry theta = 0
            div = sum(self._grad(raw * (1.0 - raw) * n[d])[d] for d in range(3))
            lap = self._lap(raw)
            phi = raw
            if p["phi_correction"]:
                mid = (raw > 0.5) & (raw < 0.9)
                if self.fluid is not None:
                    mid &= self.fluid
                cnt = mid.sum()
                if int(cnt):
                    corr = (self.sum0 - self._sum(raw)) / cnt
                    phi = torch.where(mid, raw + corr, raw)
            if dr:
                rho = p["rho_r"] * phi + (1.0 - phi) * p["rho_b"]
                f = [rho * c for c in f]
            chem = 4.0 * self.beta * phi * (phi - 1.0) * (phi - 0.5) - self.kappa * lap
            f = [a + chem * b for a, b in zip(f, gf)]
            if p["repulsive_flux"]:
                f = [a + (b * rho).clamp(-1e-3, 1e-3) * rho for a, b in zip(f, self._repulsion(phi, raw))]
            nu = (p["rho_r"] * p["visc1"] * phi + (1.0 - phi) * p["visc2"] * p["rho_b"]) / rho
        else:
            nu = one * p["visc1"]
        om = 1.0 / (3.0 * nu + 0.5)
        u, v, w = u.clone(), v.clone(), w.clone()
        if dr:
            drho = p["rho_r"] - p["rho_b"]
            gr = [drho * c for c in gf]
            mask = 4.0 * phi * (1.0 - phi)
            f = [a - mask * P / 3.0 * b for a, b in zip(f, gr)]
        tf = [c.clone() for c in f]

        def stress(pi, a, b, c):
            q = [s - t for s, t in zip(pi, (a * a, b * b, c * c, a * b, a * c, b * c))]
            return (q[0] * gr[0] + q[3] * gr[1] + q[4] * gr[2], q[1] * gr[1] + q[3] * gr[0] + q[5] * gr[2],
                    q[2] * gr[2] + q[4] * gr[0] + q[5] * gr[1])

        if dr:
            cv = mask * nu * om * 3.0
            f = [a - cv * b for a, b in zip(f, stress(pi, *self.uold))]
        u, v, w = u + 0.5 * f[0] / rho, v + 0.5 * f[1] / rho, w + 0.5 * f[2] / rho
        if dr:
            dd = drho * (p["tau_diff"] * lap - self.sharp * div)
            den = 1.0 - 0.5 * dd / rho
            u, v, w = u / den, v / den, w / den
            tf = [a - dd * b for a, b in zip(tf, (u, v, w))]
            f = [a - dd * b for a, b in zip(f, (u, v, w))]
        add = (f[0] * u, f[1] * v, f[2] * w, 0.5 * (f[1] * u + f[0] * v), 0.5 * (f[2] * u + f[0] * w),
               0.5 * (f[2] * v + f[1] * w))
        pi = [a + b / rho for a, b in zip(pi, add)]
        if dr:
            tf = [a - cv * b for a, b in zip(tf, stress(pi, u, v, w))]
        vel = (u, v, w)
        uu = (u * u, v * v, w * w, u * v, u * w, v * w)
        neq = [a - b for a, b in zip(pi, uu)]
        if tc:
            new = phi - 0.5 * (u * gf[0] + v * gf[1] + w * gf[2]) + p["tau_diff"] * lap - self.sharp * div

        def smag(nu, rho, om):
            if not p["smagorinsky"]:
                return om
            q = neq[0] ** 2 + neq[1] ** 2 + neq[2] ** 2 + 2 * (neq[3] ** 2 + neq[4] ** 2 + neq[5] ** 2)
            c = float(np.float32(0.053) * np.float32(18.0))
            return 1.0 / (0.5 + (3 * nu + torch.sqrt((3 * nu) ** 2 + c * torch.sqrt(2.0 * q) / (rho if dr else 1.0))) / 6.0)

        # a node seen across a periodic face collides with its phi before the mass correction
        stale = None
        if corr is not None:
            rs = p["rho_r"] * raw + (1.0 - raw) * p["rho_b"] if dr else one
            ns = (p["rho_r"] * p["visc1"] * raw + (1.0 - raw) * p["visc2"] * p["rho_b"]) / rs
            stale = self._populations(P, vel, pi, [c / rs for c in tf], smag(ns, rs, 1.0 / (3.0 * ns + 0.5)))
        om_c = smag(nu, rho, om)
        F = [c / rho for c in tf]
        out = torch.zeros_like(self.mom)
        own = {}
        mine = self._populations(P, vel, pi, F, om_c)

        def take(e, h, where=None):
            x, y, z = e
            for k, a in enumerate((1, x, y, z, x * x - 1 / 3, y * y - 1 / 3, z * z - 1 / 3, x * y, x * z, y * z)):
                if a:
                    out[k] += a * h

        for e, h in mine:
            if self.fluid is not None:
                h = torch.where(self.fluid, h, torch.zeros_like(h))
                if p["bounce_back"]:
                    own[e] = h
            back = tuple(-k for k in e)
            s = _at(h, back, self.pbc, 0.0)
            if stale is not None:
                e2, h2 = next(stale)
                assert e2 == e
                s2 = torch.roll(h2, (e[2], e[1], e[0]), dims=(0, 1, 2))
                for axis, k in zip((2, 1, 0), e):
                    if k:
                        at = 0 if k > 0 else s.shape[axis] - 1
                        s.select(axis, at).copy_(s2.select(axis, at))
            take(e, s)
        if self.fluid is not None:
            o = 1.0 - om_c
            for e in self.links[1:]:
                x, y, z = e
                solid = (self.isf == -1) & (_at(self.isf, tuple(-k for k in e), self.pbc, 1) == 0)
                wl = _WEIGHT[p["lattice"]][x * x + y * y + z * z]
                if p["bounce_back"]:
                    h = own[tuple(-k for k in e)]
                    take(e, torch.where(solid, h, torch.zeros_like(h)))
                    continue
                h = wl * P + o * wl * 4.5 * ((x * x - 1 / 3) * neq[0] + (y * y - 1 / 3) * neq[1] + (z * z - 1 / 3) * neq[2]
                                             + 2 * (x * y * neq[3] + x * z * neq[4] + y * z * neq[5]))
                take(e, torch.where(solid, h, torch.zeros_like(h)))
        if p["openbc"]:
            self._open_faces(out, P, vel, pi, om)
        self.last = dict(press=P.clone(), vel=torch.stack(vel), phi=phi)
        if self.fluid is not None:
            self.last["vel"] = torch.where(self.fluid, self.last["vel"], self.uold)
        self.mom, self.uold = out, self.last["vel"]
        if tc:
            if self.fluid is not None:
                new = torch.where(self.fluid, new, self.other)
                if self.pending is not None:
                    new[self.wk, self.wj, self.wi] = self.pending
                self.pending = ghost
                self.last["phi"] = phi.clone()
                self.last["phi"][self.wk, self.wj, self.wi] = ghost
            self.phi, self.other = new, raw
        self.n += 1

    def _open_faces(self, out, P, vel, pi, om):
        """The wall links of the nodes next to each open face take the face's populations instead of bounce-back's."""
        p = self.p
        u, v, w = vel
        uu = (u * u, v * v, w * w, u * v, u * w, v * w)
        pq = [a - b - (P / 3.0 if k < 3 else 0.0) for k, (a, b) in enumerate(zip(pi, uu))]
        shape = self.isf.shape
        for axis in range(3):
            if self.pbc[axis]:
                continue
            for side in range(2):
                sl = [slice(1, n - 1) for n in shape]
                sl[2 - axis] = slice(shape[2 - axis] - 2, shape[2 - axis] - 1) if side else slice(1, 2)
                sl = tuple(sl)
                kind = p["openbc_type"][axis][side]
                pb, vb = P[sl], [c[sl] for c in vel]
                if kind == 1:
                    pb = torch.full_like(pb, p["openbc_press"][axis][side])
                elif kind != 2:
                    vb = [torch.zeros_like(pb) for _ in range(3)]
                o = 1.0 - om[sl]
                half = 1.5 * (vb[0] ** 2 + vb[1] ** 2 + vb[2] ** 2)
                for e in self.links[1:]:
                    x, y, z = e
                    hit = ((self.isf == -1) & (_at(self.isf, tuple(-k for k in e), self.pbc, 1) == 0))[sl]
                    wl = _WEIGHT[p["lattice"]][x * x + y * y + z * z]
                    q = [c[sl] for c in pq]
                    qn = 4.5 * ((x * x - 1 / 3) * q[0] + (y * y - 1 / 3) * q[1] + (z * z - 1 / 3) * q[2]
                                + 2 * (x * y * q[3] + x * z * q[4] + y * z * q[5]))
                    fo = wl * P[sl] + o * wl * qn
                    uc = 3.0 * (vb[0] * x + vb[1] * y + vb[2] * z)
                    fn = wl * (pb + uc + 0.5 * uc * uc - half) + o * wl * qn
                    zero = torch.zeros_like(fo)
                    fo, fn = torch.where(hit, fo, zero), torch.where(hit, fn, zero)
                    cc = (1, x, y, z, x * x, y * y, z * z, x * y, x * z, y * z)
                    for k in range(10):
                        out[(k,) + sl] += cc[k] * (fn - fo) - (fn / 3.0 if 4 <= k < 7 else 0.0)

    def sums(self):
        t = [self.phi if self.tc else None] + list(self.mom[0:4])
        return np.array([0.0 if c is None else float(self._sum(c)) for c in t])


def _exact_run(p, isf, mom, phi, steps):
    e = _Exact(p, isf, mom, phi)
    for _ in range(steps):
        e.step()
    return e


def exact(case, seed):
    c = case
    with torch.no_grad():
        if c["kind"] == "server":
            out = []
            for one, sd in _solves(c, seed):
                p, isf, mom, phi = _inputs(one, sd)
                e = _exact_run(p, isf, mom, phi, c["steps"])
                out.append((e.mom, e.phi))
            return out
        p, isf, mom, phi = _inputs(c, seed)
        e = _Exact(p, isf, mom, phi)
        if c["kind"] == "handover":
            for _ in range(c["steps"]):
                e.step()
            return {"press": e.mom[0], "vel": e.mom[1:4], "pi": e.mom[4:], "phi": e.phi, "uold": e.uold}
        for _ in range(c["steps"] // 2):
            e.step()
        sums = e.sums()
        for _ in range(c["steps"] - c["steps"] // 2):
            e.step()
        rho = e.last["press"] if not e.tc else e.last["phi"]
        return {"sums": sums, "rho": rho, "vel": torch.movedim(e.last["vel"], 0, -1), "press": e.last["press"]}
