"""The work that a user of this framework has it do, as cases to be timed.

Kinds (a case's "kind") and the public entry points behind them:

  arrays   api.update_e / update_h / update_pbc_* on contiguous tensors: the NumPy-shaped functions
  fields   Fields + Core + Pml + IncidentDirect, the KEMP-shaped objects: update_e() and update_h() per step
  yee      YeeSolver.step(n): PEC or CPML, optionally with a Drude box or a TFSF plane wave
  symp     SymplecticSolver.step(n): 4th order, stage-wise CPML
  batch    BatchSolver.run_graph(n): ragged independent grids in one captured graph
  adjoint  fdtd_run(ce, engine) and its backward: monitors and dL/dCE

Initial fields are seeded noise of amplitude 0.1, permittivity is piecewise
constant (blocks of 8 cells, eps_r in [1, 12]), sources are Gaussian-modulated
sines: every array holds values as a simulation in progress does.
"""
import math

import numpy as np
import torch

from fdtd_accelerate_gb300 import BatchSolver, YeeAdjoint, YeeSolver, api, fdtd_run
from fdtd_accelerate_gb300.drude import DrudeAde
from fdtd_accelerate_gb300.fields import Core, Fields, IncidentDirect, Pml
from fdtd_accelerate_gb300.symplectic import SymplecticSolver
from fdtd_accelerate_gb300.tfsf import Tfsf

DEV = "cuda"
EH = ("ex", "ey", "ez", "hx", "hy", "hz")


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest use of the NumPy-shaped functions: a teaching-size box with periodic planes, one step a call
        {"name": "arrays_40", "kind": "arrays", "nx": 40, "ny": 40, "nz": 40, "pbc": "xy", "steps": 1},
        # a KEMP program on the grid of the reference's 250x250x320 CUDA example (15-cell layer): one step a call,
        # as a program does that looks at its fields between the steps
        {"name": "fields_cpml_250", "kind": "fields", "nx": 250, "ny": 250, "nz": 320, "npml": 15, "steps": 1},
        # the smallest fused simulation, stepped one step at a time: latency and launches
        {"name": "yee_cpml_48_step", "kind": "yee", "nx": 48, "ny": 48, "nz": 48, "npml": 8, "steps": 1},
        # the plain 128^3 workload of bench.py (PEC walls, a point source)
        {"name": "yee_plain_128", "kind": "yee", "nx": 128, "ny": 128, "nz": 128, "npml": 0, "steps": 100},
        # an ordinary absorbing grid with odd extents in every axis
        {"name": "yee_cpml_odd", "kind": "yee", "nx": 203, "ny": 331, "nz": 157, "npml": 10, "steps": 20},
        # the default workload of bench.py: the largest
        {"name": "yee_cpml_1024", "kind": "yee", "nx": 1024, "ny": 1024, "nz": 512, "npml": 12, "steps": 10},
        # a metal: Drude box in the middle half of an absorbing grid
        {"name": "yee_drude_256", "kind": "yee", "nx": 256, "ny": 256, "nz": 256, "npml": 12, "drude": True, "steps": 10},
        # scattering: a plane wave on a total-field box
        {"name": "yee_tfsf_256", "kind": "yee", "nx": 256, "ny": 256, "nz": 256, "npml": 12, "tfsf": True, "steps": 10},
        # the 4th-order workload of bench.py
        {"name": "symp_cpml_512", "kind": "symp", "nx": 512, "ny": 512, "nz": 512, "npml": 10, "steps": 4},
        # 4th order at an ordinary size with odd extents
        {"name": "symp_cpml_odd", "kind": "symp", "nx": 150, "ny": 171, "nz": 163, "npml": 8, "steps": 4},
        # the batched workload of bench.py: 64 ragged grids, steps in one graph
        {"name": "batch_64", "kind": "batch", "sims": 64, "low": 32, "high": 192, "mult": 16, "grids": 20261204, "npml": 8,
         "steps": 20},
        # the adjoint workload's grid, with fewer steps: forward, backward, gradient in the design region
        {"name": "adjoint_256", "kind": "adjoint", "nx": 256, "ny": 256, "nz": 128, "npml": 12, "region": True,
         "steps": 96, "segment": 32},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["arrays", "fields", "yee", "yee", "yee", "symp", "batch", "adjoint"])
    if kind == "arrays":
        return {"kind": kind, "nx": size(24, 320), "ny": size(24, 320), "nz": size(24, 320),
                "pbc": rng.choice(["", "z", "xy", "xyz"]), "steps": rng.randint(1, 4)}
    if kind == "fields":
        return {"kind": kind, "nx": size(40, 320), "ny": size(40, 320), "nz": size(40, 320), "npml": rng.randint(6, 15),
                "steps": rng.randint(1, 4)}
    if kind == "yee":
        c = {"kind": kind, "nx": size(40, 700), "ny": size(40, 700), "nz": size(40, 500),
             "npml": rng.choice([0, 6, 8, 10, 12, 15]), "steps": rng.choice([1, 2, 3, 7, 10, 20])}
        extra = rng.choice(["", "", "", "drude", "tfsf"])
        if extra and min(c["nx"], c["ny"], c["nz"]) >= 4 * c["npml"] + 24:
            c[extra] = True
        return c
    if kind == "symp":
        nz = size(40, 400)
        return {"kind": kind, "nx": size(40, 400), "ny": size(40, 400), "nz": nz if rng.random() < 0.4 else nz // 4 * 4,
                "npml": rng.choice([0, 6, 8, 10]), "steps": rng.randint(1, 5)}
    if kind == "batch":
        return {"kind": kind, "sims": size(3, 64), "low": 24, "high": rng.choice([64, 96, 160]), "mult": rng.choice([1, 4, 16]),
                "grids": rng.randint(1, 10 ** 6), "npml": rng.randint(4, 8), "steps": 2 * rng.randint(1, 10)}
    return {"kind": kind, "nx": size(48, 224), "ny": size(48, 224), "nz": size(48, 128), "npml": rng.choice([0, 6, 8, 12]),
            "region": rng.random() < 0.5, "steps": rng.randint(20, 80), "segment": rng.choice([8, 16, 25])}


def batch_shapes(case):
    rng = np.random.default_rng(case["grids"])
    sizes = range(max(case["low"], 2 * case["npml"] + 4) // case["mult"] * case["mult"], case["high"] + 1, case["mult"])
    sizes = [s for s in sizes if s >= 2 * case["npml"] + 4]
    return [tuple(int(rng.choice(sizes)) for _ in range(3)) for _ in range(case["sims"])]


def shape_of(case):
    return (case["nx"], case["ny"], case["nz"])


# ------------------------------------------------------------------ inputs
def noise(shape, gen, amp=0.1):
    return torch.randn(shape, generator=gen, device=DEV, dtype=torch.float32).mul_(amp)


def inputs(shape, seed):
    """Six field arrays and three eps_r arrays, from the seed alone."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    f = [noise(shape, gen) for _ in range(6)]
    eps = []
    for _ in range(3):
        coarse = torch.rand([(n + 7) // 8 for n in shape], generator=gen, device=DEV).mul_(11.0).add_(1.0)
        for a in range(3):
            coarse = coarse.repeat_interleave(8, dim=a).narrow(a, 0, shape[a])
        eps.append(coarse.contiguous())
    return f, eps


def pulse(t, t0=40.0):
    return np.sin(2.0 * math.pi * 0.05 * t) * np.exp(-0.5 * ((t - t0) / 30.0) ** 2)


def dipoles(shape, npml, seed, count=6):
    """(component, point, t0) of the soft sources."""
    rng = np.random.default_rng(seed)
    return [(("ex", "ey", "ez")[int(rng.integers(0, 3))],
             tuple(int(rng.integers(min(npml + 2, n // 2), max(n - npml - 2, n // 2 + 1))) for n in shape),
             float(rng.uniform(20, 60))) for _ in range(count)]


def source_list(shape, npml, seed, count=6):
    t = np.arange(201, dtype=np.float64)
    return [(c, p, pulse(t, t0)) for c, p, t0 in dipoles(shape, npml, seed, count)]


def middle(shape, share):
    """A centred box of `share` of each extent: lower corner and size."""
    size = [max(4, int(n * share)) for n in shape]
    return [(n - s) // 2 for n, s in zip(shape, size)], size


def probes(shape, seed):
    rng = np.random.default_rng(seed + 1)
    lo, size = middle(shape, 0.5)
    return [("ez", tuple(int(rng.integers(a, a + s)) for a, s in zip(lo, size))) for _ in range(16)]


# ----------------------------------------------------------------- prepare
def yee_solver(shape, npml, seed, case=()):
    f, eps = inputs(shape, seed)
    ce = [0.5 / e for e in eps]
    extra = {}
    if "drude" in case:
        lo, size = middle(shape, 0.5)
        extra["drude"] = DrudeAde(shape, lo, size, device=DEV)
        extra["drude"].set_coeff(0.12, 0.02)
    if "tfsf" in case:
        lo, size = middle(shape, 0.5)
        extra["tfsf"] = Tfsf(shape, lo, [a + s for a, s in zip(lo, size)], wavelength=24.0, steps=256, device=DEV)
    s = YeeSolver(shape, ce=ce, npml=npml, sources=source_list(shape, npml, seed), device=DEV, **extra)
    s.set_fields(**dict(zip(EH, f)))
    s.plan()
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "arrays":
        f, eps = inputs(shape_of(case), seed)
        return {"case": case, "f": f, "ce": [0.5 / e for e in eps]}
    if kind == "fields":
        f, eps = inputs(shape_of(case), seed)
        F = Fields(*shape_of(case), coeff_use="e", device=DEV)
        F.set_ehs(*f)
        F.set_ces(*[0.5 / e for e in eps])
        Core(F)
        Pml(F, ("+-", "+-", "+-"), npml=case["npml"])
        centre = tuple(n // 2 for n in shape_of(case))
        IncidentDirect(F, "ez", centre, centre, lambda t: float(pulse(t)))
        return {"case": case, "F": F}
    if kind == "yee":
        return {"case": case, "s": yee_solver(shape_of(case), case["npml"], seed, case)}
    if kind == "symp":
        f, eps = inputs(shape_of(case), seed)
        centre = tuple(n // 2 for n in shape_of(case))
        s = SymplecticSolver(shape_of(case), ce=[0.743 / 24.0 / e for e in eps], npml=case["npml"],
                             sources=[("ez", centre, lambda t: float(pulse(t)))], device=DEV, max_steps=case["steps"] + 2)
        s.set_fields(**dict(zip(EH, f)))
        return {"case": case, "s": s}
    if kind == "batch":
        b = BatchSolver([yee_solver(sh, case["npml"], seed * 1000 + q) for q, sh in enumerate(batch_shapes(case))])
        b.capture(case["steps"])
        return {"case": case, "b": b}
    shape = shape_of(case)
    _, eps = inputs(shape, seed)
    lo, size = middle(shape, 0.5)
    region = tuple(slice(a, a + n) for a, n in zip(lo, size)) if case["region"] else None
    eng = YeeAdjoint(shape, case["steps"], npml=case["npml"], sources=source_list(shape, case["npml"], seed),
                     monitors=probes(shape, seed), segment=case["segment"], grad_region=region, device=DEV)
    ce = torch.stack([0.5 / e for e in eps]).requires_grad_(True)
    return {"case": case, "eng": eng, "ce": ce}


# --------------------------------------------------------------------- run
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "arrays":
        f, ce, pbc = state["f"], state["ce"], case["pbc"]
        for _ in range(case["steps"]):
            api.update_e(*f, *ce)
            if pbc:
                api.update_pbc_e(pbc, *f[:3])
            api.update_h(*f)
            if pbc:
                api.update_pbc_h(pbc, *f[3:])
        return f
    if kind == "fields":
        F = state["F"]
        for _ in range(case["steps"]):
            F.update_e()
            F.update_h()
        return [F.get(k) for k in EH]
    if kind == "yee":
        s = state["s"]
        s.tstep = 1  # the run's own time: a pass is a run of `steps` steps from the fields at hand
        s.step(case["steps"])
        return s.fields
    if kind == "symp":
        s = state["s"]
        s.tstep = 1
        s.step(case["steps"])
        return s.fields
    if kind == "batch":
        b = state["b"]
        for s in b.solvers:
            s.tstep = 1
        b.run_graph(case["steps"])
        # 64 outputs at most: the grids' E and H arrays laid end to end, one tensor a component
        return {k: torch.cat([s.fields[k].reshape(-1) for s in b.solvers]) for k in EH}
    ce = state["ce"]
    ce.grad = None
    mon, fields = fdtd_run(ce, state["eng"])
    (mon.double() ** 2).sum().backward()
    return {"mon": mon.detach(), "fields": fields.detach(), "grad": ce.grad}


# -------------------------------------------------------------------- work
def slab_cells(shape, npml):
    n = shape[0] * shape[1] * shape[2]
    return sum(2 * npml * (n // m) for m in shape)


def work(case):
    """Each input (fields, psi, coefficients) read once and each output written once in a pass; 30 operations a
    cell and step for the 2nd-order curls, 4 x (E + H) + H stages of 27 operations a component for the 4th-order ones."""
    kind, steps = case["kind"], case["steps"]
    shapes = batch_shapes(case) if kind == "batch" else [shape_of(case)]
    npml = case.get("npml", 0)
    cells = sum(a * b * c for a, b, c in shapes)
    slabs = sum(slab_cells(s, npml) for s in shapes)
    state = 60 * cells + 32 * slabs
    if kind == "symp":
        return {"bytes": state, "flops": 9 * 33 * cells * steps}
    if kind == "adjoint":
        # coefficients in, gradient, monitors and final fields out; the E increment of every step is needed again by the
        # reverse step: forward and reverse
        return {"bytes": (12 + 12 + 24) * cells, "flops": (30 + 48) * cells * steps}
    if case.get("drude"):
        _, size = middle(shapes[0], 0.5)
        state += 48 * size[0] * size[1] * size[2]
    if kind == "batch":
        state += 48 * cells  # the outputs laid end to end
    return {"bytes": state, "flops": 30 * cells * steps}


# ------------------------------------------------------------------- exact
def cpml64(n, P, dt, e):
    """b, a, 1/kappa - 1 along one axis of n nodes (FP64, zero off the layer): m = 4, R = 1e-8, kappa_max = 5,
    alpha_max = 0.05; E nodes 1..P and n-P-1..n-2, H nodes 1..P and n-P..n-1."""
    out = [np.zeros(n) for _ in range(3)]
    if P:
        q = np.arange(P, dtype=np.float64)
        front, back = (P - q - 0.5, q + 0.5) if e else (P - q, q + 1.0)
        first = n - P - 1 if e else n - P
        for at, depth in ((1, front), (first, back)):
            x = depth / P
            sig = -5.0 * math.log(1e-8) / (2.0 * P) * x ** 4
            kap, alp = 1.0 + 4.0 * x ** 4, 0.05 * (1.0 - x)
            b = np.exp(-(sig / kap + alp) * dt)
            den = sig * kap + alp * kap * kap
            a = np.where(den > 0, sig / np.where(den > 0, den, 1.0) * (b - 1.0), 0.0)
            for o, v in zip(out, (b, a, 1.0 / kap - 1.0)):
                o[at:at + P] = v
    return [torch.from_numpy(o).to(DEV) for o in out]


class Exact:
    """The step in FP64 by plain tensor operations, out of place. order: 2 (Yee) or 4 (one symplectic stage)."""

    def __init__(self, shape, npml, order):
        self.shape, self.npml, self.order = shape, npml, order
        self.psi = {}
        self.prof = {}

    def d(self, F, a):
        """Difference along axis a at the nodes that E / H updates: 0..n-2 / 1..n-1, or 1..n-3 / 2..n-2."""
        n = self.shape[a]
        if self.order == 2:
            return F.narrow(a, 1, n - 1) - F.narrow(a, 0, n - 1)
        return 27.0 * (F.narrow(a, 2, n - 3) - F.narrow(a, 1, n - 3)) - (F.narrow(a, 3, n - 3) - F.narrow(a, 0, n - 3))

    def first(self, e):
        return (0 if e else 1) if self.order == 2 else (1 if e else 2)

    def term(self, F, comp, a, e, dt):
        """The difference with its CPML terms, cut to the nodes that component `comp` updates on the other axis."""
        D = self.d(F, a)
        other = 3 - comp - a
        m, at = D.shape[a], self.first(e)
        D = D.narrow(other, at, self.shape[other] - 1 if self.order == 2 else self.shape[other] - 3)
        if self.npml:
            key = (a, e, dt)
            if key not in self.prof:
                view = [1, 1, 1]
                view[a] = m
                self.prof[key] = [v[at:at + m].reshape(view) for v in cpml64(self.shape[a], self.npml, dt, e)]
            b, c, k = self.prof[key]
            psi = self.psi.get((comp, a, e), 0.0)
            psi = b * psi + c * D
            self.psi[(comp, a, e)] = psi
            D = D + (k * D + psi)
        return D

    def update(self, E, H, e, coef, dt):
        """E (e) or H updated from the other family: coef a number, or one array a component."""
        src = H if e else E
        out = []
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3   # component c: + d(F_v)/d(u) - d(F_u)/d(v)
            D = self.term(src[v], c, u, e, dt) - self.term(src[u], c, v, e, dt)
            at = self.first(e)
            k = coef if isinstance(coef, float) else coef[c]
            full = (E if e else H)[c].clone()
            for ax in (u, v):
                if not isinstance(k, float):
                    k = k.narrow(ax, at, D.shape[ax])
            part = full.narrow(u, at, D.shape[u]).narrow(v, at, D.shape[v])
            part.add_(k * D if e else -(k * D))
            out.append(full)
        return out


def add_sources(E, src, t):
    for comp, p, amp in src:
        if t < len(amp):
            E["xyz".index(comp[1])][p] += float(np.float32(amp[t]))


def yee64(f, ce, shape, npml, steps, src, drude=False, pbc="", mon=None):
    X = Exact(shape, npml, 2)
    E, H = f[:3], f[3:]
    if drude:
        lo, size = middle(shape, 0.5)
        box = tuple(slice(a, a + s) for a, s in zip(lo, size))
        wp, g, dt = (float(np.float32(v)) for v in (0.12, 0.02, 0.5))
        cja, cjb = (2 - g * dt) / (2 + g * dt), 4 * (dt * wp) ** 2 / (2 + g * dt)
        J = [0.0] * 3
    rows = []
    for t in range(1, steps + 1):
        E = X.update(E, H, True, ce, 0.5)
        if drude:
            for c in range(3):
                v = E[c][box]
                v -= ce[c][box] * J[c]
                J[c] = cja * J[c] + cjb * v
        for q, n in (("x", 0), ("y", 1), ("z", 2)):
            if q in pbc:
                for c in ((n + 1) % 3, (n + 2) % 3):
                    E[c].select(n, -1).copy_(E[c].select(n, 0))
        add_sources(E, src, t)
        H = X.update(E, H, False, 0.5, 0.5)
        for q, n in (("x", 0), ("y", 1), ("z", 2)):
            if q in pbc:
                for c in ((n + 1) % 3, (n + 2) % 3):
                    H[c].select(n, 0).copy_(H[c].select(n, -1))
        if mon:
            rows.append(torch.stack([(E + H)[EH.index(c)][p] for c, p in mon]))
    return E + H, rows


def symp64(f, ce, shape, npml, steps, src):
    c1, c2, c3, d1, d2, S = 0.17399689146541, -0.12038504121430, 0.89277629949778, 0.62337932451322, -0.12337932451322, 0.743
    X = Exact(shape, npml, 4)
    E, H = f[:3], f[3:]
    for t in range(1, steps + 1):
        for sn, (c, d) in enumerate(((c1, d1), (c2, d2), (c3, d2), (c2, d1))):
            H = X.update(E, H, False, c * S / 24.0, c * S)
            E = X.update(E, H, True, [d * v for v in ce], d * S)
            for comp, p, fn in src:
                E["xyz".index(comp[1])][p] += float(np.float32(fn(t + sn / 5.0)))
        H = X.update(E, H, False, c1 * S / 24.0, c1 * S)
    return E + H


def adjoint64(case, seed):
    """Gradient in FP64 by autograd, segment by segment from stored states."""
    shape, npml, steps = shape_of(case), case["npml"], case["steps"]
    ce = [(0.5 / e).double() for e in inputs(shape, seed)[1]]
    src, mon = source_list(shape, npml, seed), probes(shape, seed)

    def segment(state, psi, ce, t0, t1):
        X = Exact(shape, npml, 2)
        X.psi = dict(psi)
        E, H, rows = list(state[:3]), list(state[3:]), []
        for t in range(t0 + 1, t1 + 1):
            E = X.update(E, H, True, ce, 0.5)
            add_sources(E, src, t)
            H = X.update(E, H, False, 0.5, 0.5)
            rows.append(torch.stack([(E + H)[EH.index(c)][p] for c, p in mon]))
        return E + H, X.psi, rows

    zero = torch.zeros(shape, dtype=torch.float64, device=DEV)
    state, psi, saved, rows, cuts = [zero] * 6, {}, [], [], list(range(0, steps, 8)) + [steps]
    with torch.no_grad():
        for t0, t1 in zip(cuts, cuts[1:]):
            saved.append((state, psi))
            state, psi, r = segment(state, psi, ce, t0, t1)
            rows += r
    final = torch.stack(state)
    lam, lpsi, grad = None, None, [torch.zeros_like(v) for v in ce]
    for (state, psi), t0, t1 in reversed(list(zip(saved, cuts, cuts[1:]))):
        leaf = [v.clone().requires_grad_(True) for v in state]
        pleaf = {k: v.clone().requires_grad_(True) for k, v in psi.items()}
        cleaf = [v.clone().requires_grad_(True) for v in ce]
        out, pout, r = segment(leaf, pleaf, cleaf, t0, t1)
        outs, grads = [(torch.stack(r) ** 2).sum()], [None]
        if lam is not None:
            outs += [o for o, g in zip(out, lam) if g is not None]
            grads += [g for g in lam if g is not None]
            outs += [pout[k] for k in pout if lpsi.get(k) is not None]
            grads += [lpsi[k] for k in pout if lpsi.get(k) is not None]
        keys = list(pleaf)
        got = torch.autograd.grad(outs, leaf + [pleaf[k] for k in keys] + cleaf, grads, allow_unused=True)
        lam, lpsi = got[:6], dict(zip(keys, got[6:6 + len(keys)]))
        grad = [g + (v if v is not None else 0.0) for g, v in zip(grad, got[6 + len(keys):])]
    grad = torch.stack(grad)
    if case["region"]:
        keep = torch.zeros(shape, dtype=torch.float64, device=DEV)
        lo, size = middle(shape, 0.5)
        keep[tuple(slice(a, a + n) for a, n in zip(lo, size))] = 1.0
        grad = grad * keep
    return {"mon": torch.stack(rows), "fields": final, "grad": grad}


def exact(case, seed):
    kind, steps = case["kind"], case["steps"]
    if case.get("tfsf"):
        return None  # the 1-D incident grid is the framework's own definition of the wave
    if kind == "adjoint":
        return adjoint64(case, seed)
    with torch.no_grad():
        if kind == "batch":
            parts = []
            for q, sh in enumerate(batch_shapes(case)):
                f, eps = inputs(sh, seed * 1000 + q)
                parts.append(yee64([v.double() for v in f], [(0.5 / e).double() for e in eps], sh, case["npml"], steps,
                                   source_list(sh, case["npml"], seed * 1000 + q))[0])
            return {k: torch.cat([p[n].reshape(-1) for p in parts]) for n, k in enumerate(EH)}
        shape = shape_of(case)
        f, eps = inputs(shape, seed)
        f = [v.double() for v in f]
        centre = tuple(n // 2 for n in shape)
        if kind == "symp":
            out = symp64(f, [(0.743 / 24.0 / e).double() for e in eps], shape, case["npml"], steps, [("ez", centre, pulse)])
            return dict(zip(EH, out))
        ce = [(0.5 / e).double() for e in eps]
        del eps
        if kind == "arrays":
            return yee64(f, ce, shape, 0, steps, [], pbc=case["pbc"])[0]
        if kind == "fields":
            src = [("ez", centre, pulse(np.arange(steps + 1, dtype=np.float64)))]
            return yee64(f, ce, shape, case["npml"], steps, src)[0]
        out = yee64(f, ce, shape, case["npml"], steps, source_list(shape, case["npml"], seed), drude="drude" in case)[0]
        return dict(zip(EH, out))
