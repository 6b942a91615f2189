"""Performance cases of the MUSCL-Hancock step: what users of the framework run.

listed() gives the cases, draw(rng) more of the same ranges.  prepare(case,
seed) makes the inputs on the GPU and the handle a program keeps; run(state)
is one pass through the public entry points; exact(case, seed) computes the
same outputs with plain torch in 64 bits.  A pass of the time-loop cases is
what a driver does between two outputs: the state goes in (hcl_set_state), a
number of CFL steps run (hcl_run), the state comes out (hcl_get_state).
"""
import functools
import math

import numpy as np
import torch

from heraclespp_b200 import Domain, Ensemble

CFL = 0.4
BC = {"P": "Periodic", "N": "NullGradient", "R": "Reflexive"}
G_NEWTON = 6.6743015e-11


def _case(name, **kw):
    """A case with every key: sizes n0 x n1 x n2 (1 on unused dimensions),
    `bc` one letter per face (x low, x high, y low, ...), `flow` the initial
    state, `steps` time steps of a pass (0: to t = 0.2)."""
    c = dict(name=name, kind="run", ndim=2, n0=1, n1=1, n2=1, steps=1, precision="fp64", limiter="VanLeer",
             riemann="HLLC", bc="PPPPPP", geometry="Cartesian", gravity="Uniform", gz=0.0, central_mass=0.0, nfx=0,
             flow="shear", gamma=1.4, every=0, problems=0)
    c.update(kw)
    return c


FAMILIES = [
    # The smallest runs: a 1-D shock tube of 1024 cells taken to t = 0.2 (the
    # method's standard check), where the latency of a step is everything.
    _case("sod1d_1024_fp64", ndim=1, n0=1024, steps=0, limiter="Minmod", bc="NNPPPP", flow="sod"),
    # A small odd 2-D shear layer in FP32-mixed, as in parameter scans and
    # tutorials: below one wave of the card.
    _case("shear2d_200x136_mixed", n0=200, n1=136, steps=120, precision="fp32_mixed"),
    # Kelvin-Helmholtz 2048^2, FP32-mixed: the benchmark's headline.
    _case("shear2d_2048_mixed", n0=2048, n1=2048, steps=60, precision="fp32_mixed"),
    # The same grid in the plain FP64 that reproduces the reference's bits.
    _case("shear2d_2048_fp64", n0=2048, n1=2048, steps=6),
    # Four-quadrant outflow problem on ragged sizes in fast FP64.
    _case("quadrant2d_1333x1001_fast64", n0=1333, n1=1001, steps=12, precision="fp64_fast", limiter="Minmod",
          bc="NNNNPP", flow="quadrant"),
    # Ragged stratified 2-D run with walls, gravity and two passive scalars
    # (mass fractions of a mixing layer), FP32-mixed.
    _case("strat2d_1500x701_fx2_mixed", n0=1500, n1=701, steps=40, precision="fp32_mixed", bc="PPRRPP", gz=-0.1,
          flow="strat", nfx=2),
    # Rayleigh-Taylor 256^2 x 512 in FP32-mixed: the largest grid.
    _case("strat3d_256x256x512_mixed", ndim=3, n0=256, n1=256, n2=512, steps=8, precision="fp32_mixed",
          limiter="Minmod", riemann="HLL", bc="PPPPRR", gz=-0.1, flow="strat"),
    # Rayleigh-Taylor at half the resolution in the reference's FP64.
    _case("strat3d_128x128x256_fp64", ndim=3, n0=128, n1=128, n2=256, steps=4, limiter="Minmod", riemann="HLL",
          bc="PPPPRR", gz=-0.1, flow="strat"),
    # A stellar shell on a spherical wedge with gravity from the enclosed mass
    # and one mass fraction: the science runs of the reference.
    _case("shell3d_96x64x50_fp64", ndim=3, n0=96, n1=64, n2=50, steps=10, bc="RNRRPP", geometry="Spherical",
          gravity="Internal_mass", central_mass=1e9, nfx=1, flow="shell"),
    # A host code that keeps its own loop and arrays and replaces one plugin
    # after another: every stage of the step through its own entry point.
    _case("stages3d_120x100x70_fp64", kind="stages", ndim=3, n0=120, n1=100, n2=70, steps=3, bc="PPPPRR", gz=-0.1,
          flow="strat"),
    # Gradient of a vortex run with respect to its initial state
    # (checkpointed forward and reverse sweep), in FP64.
    _case("vortex2d_adjoint_512_fp64", kind="adjoint", n0=512, n1=512, steps=40, flow="vortex", gamma=5.0 / 3.0,
          every=16),
    # A batch of uneven four-quadrant problems stepped in one launch, and the
    # gradient of their total energy (FP32-mixed, FP32 reverse sweep).
    _case("ensemble2d_15_mixed", kind="ensemble", n0=1024, n1=1024, steps=20, precision="fp32_mixed",
          limiter="Minmod", bc="NNNNPP", flow="quadrant", every=10, problems=15),
]


def listed():
    return [dict(c) for c in FAMILIES]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of one family with sizes, limiter, solver and boundaries drawn
    over the family's range (at most the listed case's cells)."""
    c = dict(rng.choice(FAMILIES))
    del c["name"]
    c["limiter"] = rng.choice(["VanLeer", "Minmod", "VanAlbada"])
    c["riemann"] = rng.choice(["HLL", "HLLC"])
    if c["kind"] == "ensemble":
        c["problems"] = rng.randint(3, c["problems"])
        c["steps"] = rng.randint(8, 16)
        return c
    if c["ndim"] == 1:
        c["n0"] = _log_int(rng, 100, 1100)
        c["precision"] = rng.choice(["fp64", "fp64_fast"])
        return c
    if c["kind"] == "adjoint":
        c["n0"], c["n1"] = _log_int(rng, 96, 512), _log_int(rng, 96, 512)
        c["precision"] = rng.choice(["fp64", "fp32_mixed"])
        return c
    scale = 1.0 if c["n0"] * c["n1"] * c["n2"] < 10 ** 5 else rng.uniform(0.08, 1.0) ** (1.0 / c["ndim"])
    for key in ("n0", "n1", "n2")[: c["ndim"]]:
        c[key] = max(12, int(c[key] * scale * rng.uniform(0.7, 1.0)))
    if c["geometry"] == "Cartesian":
        pair = {"shear": ["PP", "NN", "RR"], "quadrant": ["NN", "RR"], "strat": ["PP"]}[c["flow"]]
        walls = rng.choice(pair)
        last = "RR" if c["flow"] == "strat" else rng.choice(pair)
        c["bc"] = (walls + last + "PP") if c["ndim"] == 2 else ("PP" + walls + last)
    return c


def work(case):
    """Bytes: the FP64 state in and out of a pass.  A step's dt depends on
    every cell of the step before, so a state that does not fit the card's
    cache (126 MB) goes through memory once per step.  A gradient also reads
    dJ/dU^N and writes dJ/dU^0.  Flops: primitives, slopes, predictor, one
    Riemann problem per face and the update, counted per cell and step; the
    reverse sweep of a step is four steps' worth."""
    nv = case["ndim"] + 2 + case["nfx"]
    flops = {1: 200, 2: 420, 3: 750}[case["ndim"]]
    steps = case["steps"] or round(0.2 * case["n0"] * 2.3 / CFL)
    if case["kind"] == "ensemble":
        cells = sum(a * b for a, b in _ensemble_sizes(case))
    else:
        cells = case["n0"] * case["n1"] * case["n2"]
    state = cells * 8 * nv
    if case["kind"] in ("adjoint", "ensemble"):
        return {"bytes": state * 4, "flops": cells * steps * flops * 5}
    return {"bytes": state * 2 * (steps if state > 126e6 else 1), "flops": cells * steps * flops}


# ---- grids, initial states, boundaries ---------------------------------------
NG = 2


def _ensemble_sizes(case):
    """Uneven sides from {128, 256, 512, 1024}, the same for every seed."""
    rng = np.random.default_rng(2024 + case["problems"])
    top = case["n0"]
    sides = [s for s in (128, 256, 512, 1024) if s <= top]
    return [(int(rng.choice(sides)), int(rng.choice(sides))) for _ in range(case["problems"])]


def _extent(case):
    if case["geometry"] == "Spherical":
        return (0.2, 0.6, 0.0), (1.2, 2.5, 1.5)
    if case["ndim"] == 3:
        return (0.0, 0.0, 0.0), (0.5, 0.5, 1.0)
    return (0.0, 0.0, 0.0), (1.0, 1.0, 1.0)


def _gvec(case):
    g = [0.0, 0.0, 0.0]
    g[case["ndim"] - 1] = case["gz"]
    return tuple(g)


def _keywords(case):
    xmin, xmax = _extent(case)
    return dict(gamma=case["gamma"], limiter=case["limiter"], riemann=case["riemann"], geometry=case["geometry"],
                gravity=case["gravity"], central_mass=case["central_mass"] or 1.0, g=_gvec(case), nfx=case["nfx"],
                bc=[BC[x] for x in case["bc"]], xmin=xmin, xmax=xmax, precision=case["precision"])


class _Mesh:
    """Node coordinates and per-cell geometry of a case (torch, FP64)."""

    def __init__(self, case, dev):
        nd = case["ndim"]
        xmin, xmax = _extent(case)
        self.nd, self.dev = nd, dev
        self.nx = [case["n0"], case["n1"], case["n2"]]
        self.ng = [NG if d < nd else 0 for d in range(3)]
        self.n = [self.nx[d] + 2 * self.ng[d] for d in range(3)]
        self.shape = (self.n[2], self.n[1], self.n[0])
        self.x, self.dx, self.xc = [], [], []
        for d in range(3):
            i = torch.arange(self.n[d] + 1, dtype=torch.float64, device=dev) - self.ng[d]
            x = xmin[d] + i * ((xmax[d] - xmin[d]) / self.nx[d])
            view = [1, 1, 1]
            view[2 - d] = -1
            self.x.append(x.view(view))
            self.dx.append((x[1:] - x[:-1]).view(view))
            self.xc.append(((x[1:] + x[:-1]) / 2).view(view))
        self.spherical = case["geometry"] == "Spherical"
        self.inner = tuple(slice(self.ng[d], self.n[d] - self.ng[d]) for d in (2, 1, 0))
        if self.spherical:
            r0, r1 = self.x[0][..., :-1], self.x[0][..., 1:]
            t0, t1 = self.x[1][:, :-1], self.x[1][:, 1:]
            dcos, dphi = torch.cos(t0) - torch.cos(t1), self.dx[2]
            self.dv = (r1 ** 3 - r0 ** 3) / 3 * dcos * dphi
            self.ds = [[r0 ** 2 * dcos * dphi, r1 ** 2 * dcos * dphi],
                       [(r1 ** 2 - r0 ** 2) / 2 * torch.sin(t0) * dphi, (r1 ** 2 - r0 ** 2) / 2 * torch.sin(t1) * dphi],
                       [r0 * self.dx[0] * self.dx[1]] * 2]
            self.rfac = (r1 - r0) / (r1 + r0)
            self.cot = torch.cos((t0 + t1) / 2) / torch.sin((t0 + t1) / 2)
            self.pfac = (torch.sin(t1) - torch.sin(t0)) / (torch.sin(t1) + torch.sin(t0))
            r = self.xc[0]
            self.width = [self.dx[0], self.dx[1] * r, self.dx[2] * r * torch.sin(self.xc[1])]
        else:
            self.dv = self.dx[0] * self.dx[1] * self.dx[2]
            self.ds = [[self.dv / self.dx[d]] * 2 for d in range(3)]
            self.width = self.dx
        self.maps = [self._map(d, case["bc"]) for d in range(nd)]

    def _map(self, d, bc):
        """Source index and normal-momentum sign of each cell along d."""
        n, nx = self.n[d], self.nx[d]
        src, sign = [], []
        for i in range(n):
            if i < NG:
                s = {"P": (i + nx, 1), "N": (NG, 1), "R": (2 * NG - 1 - i, -1)}[bc[2 * d]]
            elif i >= n - NG:
                s = {"P": (i - nx, 1), "N": (n - NG - 1, 1), "R": (2 * (n - NG) - 1 - i, -1)}[bc[2 * d + 1]]
            else:
                s = (i, 1)
            src.append(s[0])
            sign.append(s[1])
        view = [1, 1, 1]
        view[2 - d] = -1
        return (torch.tensor(src, device=self.dev),
                torch.tensor(sign, dtype=torch.float64, device=self.dev).view(view))

    def fill(self, q):
        """Ghost cells of every field of q (rho, momenta, E, scalars)."""
        out = list(q)
        for d, (src, sign) in enumerate(self.maps):
            for v in range(len(out)):
                out[v] = torch.index_select(out[v], 2 - d, src)
                if v == 1 + d:
                    out[v] = out[v] * sign
        return out


def _initial(case, mesh, seed):
    """Conserved state with ghosts: [rho, momenta..., E, scalars...].  Smooth
    seeded modes in every field (a flow some way into its run) on the flow's
    own structure, with cell noise of 1e-3."""
    nd, dev = mesh.nd, mesh.dev
    rng = np.random.default_rng([seed, case["n0"], case["n1"]])
    unit = []
    for d in range(3):
        lo, hi = _extent(case)[0][d], _extent(case)[1][d]
        unit.append((mesh.xc[d] - lo) / (hi - lo))
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(rng.integers(1 << 31)))
    X, Y, Z = unit

    def modes(amp):
        out = torch.zeros(mesh.shape, dtype=torch.float64, device=dev)
        for _ in range(4):
            k = rng.integers(1, 5, size=3)
            arg = 2 * math.pi * (int(k[0]) * X + (int(k[1]) * Y if nd > 1 else 0) + (int(k[2]) * Z if nd > 2 else 0))
            out = out + amp / 2 * float(rng.uniform(0.5, 1)) * torch.cos(arg + float(rng.uniform(0, 2 * math.pi)))
        noise = torch.rand(mesh.shape, generator=gen, dtype=torch.float64, device=dev)
        return out + 1e-3 * (2 * noise - 1)

    zero = torch.zeros(mesh.shape, dtype=torch.float64, device=dev)
    u = [zero] * nd
    top = unit[nd - 1]
    frac = (1 + modes(0.4)) / 2
    if case["flow"] == "sod":
        cut = float(rng.uniform(0.45, 0.55))
        left = X <= cut
        pl, pr, rl, rr = (float(v) for v in rng.uniform([0.95, 0.09, 0.95, 0.115], [1.05, 0.11, 1.05, 0.135]))
        rho, P = torch.where(left, rl, rr) + zero, torch.where(left, pl, pr) + zero
        return mesh.fill([rho, rho * u[0], P / (case["gamma"] - 1)])
    if case["flow"] == "shear":
        band = (Y - 0.5).abs() < 0.25
        rho, P = torch.where(band, 2.0, 1.0) + modes(0.05), 2.5 + modes(0.05)
        u[0], u[1] = torch.where(band, 0.5, -0.5) + modes(0.05), modes(0.15)
    elif case["flow"] == "quadrant":
        which = (X > 0.5).long() + 2 * (Y > 0.5).long()
        pick = [torch.tensor(rng.uniform(lo, hi, 4), device=dev)[which] for lo, hi in ((0.3, 2), (-1, 1), (-1, 1), (0.3, 2))]
        rho, P = pick[0] * (1 + modes(0.1)), pick[3] * (1 + modes(0.1))
        u[0], u[1] = pick[1] + modes(0.1), pick[2] + modes(0.1)
    elif case["flow"] == "strat":
        up = top > 0.5
        rho = torch.where(up, 2.0, 1.0) * (1 + modes(0.05))
        P = 2.5 - 0.1 * torch.where(up, 2.0, 1.0) * (top - 0.5) + modes(0.03)
        u = [modes(0.2) for _ in range(nd)]
        frac = torch.where(up, 0.9, 0.1) + modes(0.05)
    elif case["flow"] == "vortex":
        x, y = X - 0.5, Y - 0.5
        r = torch.sqrt(x * x + y * y)
        w = torch.where(r < 0.2, 5.0 + 0 * r, torch.where(r < 0.4, 2 / r - 5, 0.0 * r))
        p = torch.where(r < 0.2, 12.5 * r * r, 12.5 * r * r + 4 - 20 * r + 4 * torch.log(5 * r))
        P = 5 + torch.where(r < 0.4, p, 4 * math.log(2.0) - 2 + 0 * r) + modes(0.05)
        rho = 1 + modes(0.05)
        u[0], u[1] = -w * y + modes(0.05), w * x + modes(0.05)
    else:  # shell: density and pressure falling with the radius
        rho, P = torch.exp(-2 * X) * (1 + modes(0.1)), 1.5 * torch.exp(-2.5 * X) * (1 + modes(0.05))
        u = [modes(0.15) for _ in range(nd)]
        frac = torch.where(X < 0.4, 0.8, 0.2) + modes(0.05)
    E = P / (case["gamma"] - 1) + 0.5 * rho * sum(v * v for v in u)
    fx = [(frac * (1 - 0.3 * f)).clamp(0, 1) for f in range(case["nfx"])]
    return mesh.fill([rho] + [rho * v for v in u] + [E] + fx)


def _split(q, nd):
    """(rho, rhou, E, fx or None) as contiguous arrays of the public layout."""
    fx = torch.stack(q[nd + 2:]) if len(q) > nd + 2 else None
    return q[0].contiguous(), torch.stack(q[1:1 + nd]), q[1 + nd].contiguous(), fx


def _problems(case):
    """The ensemble's members as single cases."""
    out = []
    for a, b in _ensemble_sizes(case):
        c = dict(case)
        c.update(n0=a, n1=b, kind="run")
        out.append(c)
    return out


def _energy_adjoint(mesh):
    """dJ/dU of J = sum of E dV over the interior."""
    lam = torch.zeros((mesh.nd + 2,) + mesh.shape, dtype=torch.float64, device=mesh.dev)
    lam[(1 + mesh.nd,) + mesh.inner] = mesh.dv.expand(mesh.shape)[mesh.inner]
    return lam


def _objective_adjoint(case, mesh, seed):
    """dJ/dU at the end for J = 0.5 |rho - target|^2 is a field like the
    density's own variations: seeded modes, on the density plane."""
    rng = np.random.default_rng([seed, 77])
    lam = torch.zeros((mesh.nd + 2,) + mesh.shape, dtype=torch.float64, device=mesh.dev)
    lo, hi = _extent(case)
    for _ in range(3):
        k = rng.integers(1, 6, size=2)
        X, Y = (mesh.xc[0] - lo[0]) / (hi[0] - lo[0]), (mesh.xc[1] - lo[1]) / (hi[1] - lo[1])
        term = float(rng.uniform(0.01, 0.03)) * torch.cos(2 * math.pi * (int(k[0]) * X + int(k[1]) * Y))
        lam[(0,) + mesh.inner] += term.expand(mesh.shape)[mesh.inner]
    return lam


# ---- the measured passes --------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda", 0)
    if case["kind"] == "ensemble":
        members = _problems(case)
        sizes = [dict(nx=[m["n0"], m["n1"]], **_keywords(m)) for m in members]
        st = {"case": case, "handle": Ensemble(sizes), "init": [], "lam": [], "out": [], "grad": []}
        for p, m in enumerate(members):
            mesh = _Mesh(m, dev)
            st["init"].append(_split(_initial(m, mesh, 1000 * seed + p), 2)[:3])
            st["lam"].append(_energy_adjoint(mesh))
            st["out"].append(tuple(torch.empty_like(t) for t in st["init"][-1]))
            st["grad"].append(torch.empty_like(st["lam"][-1]))
        torch.cuda.synchronize()
        return st
    nd = case["ndim"]
    mesh = _Mesh(case, dev)
    rho, rhou, E, fx = _split(_initial(case, mesh, seed), nd)
    nx = [case["n0"], case["n1"], case["n2"]][:nd]
    st = {"case": case, "handle": Domain(nd, nx, **_keywords(case)), "init": (rho, rhou, E, fx),
          "out": [torch.empty_like(t) for t in (rho, rhou, E)], "fx": None if fx is None else torch.empty_like(fx)}
    if case["kind"] == "adjoint":
        st["lam"] = _objective_adjoint(case, mesh, seed)
        st["grad"] = torch.empty_like(st["lam"])
    if case["kind"] == "stages":
        def new(*lead):
            return torch.empty(tuple(lead) + mesh.shape, dtype=torch.float64, device=dev)

        st["stream"] = torch.cuda.Stream(dev)
        st["cur"] = [new(), new(nd), new()]
        st["new"] = [new(), new(nd), new()]
        st["prim"] = [new(nd), new()]
        st["rec"] = [new(nd, 2), new(nd, nd, 2), new(nd, 2)]
    torch.cuda.synchronize()
    return st


def run(state):
    return {"run": _run_loop, "stages": _run_stages, "adjoint": _run_adjoint,
            "ensemble": _run_ensemble}[state["case"]["kind"]](state)


def _run_loop(st):
    c, d = st["case"], st["handle"]
    rho, rhou, E, fx = st["init"]
    d.set_state(rho, rhou, E, fx=fx, device=True)
    if c["steps"]:
        d.run(cfl=CFL, nsteps=c["steps"])
    else:
        d.run(cfl=CFL, t_end=0.2)
    out = d.get_state(out=tuple(st["out"]), device=True, fx=st["fx"])
    return list(out) + ([] if fx is None else [st["fx"]])


def _run_stages(st):
    """The reference's loop with each plugin call replaced by its entry point."""
    d, ng, s = st["handle"], NG, st["stream"]
    s.wait_stream(torch.cuda.current_stream())
    raw = s.cuda_stream
    cur, new, (u, P), rec = st["cur"], st["new"], st["prim"], st["rec"]
    with torch.cuda.stream(s):
        for a, b in zip(cur, st["init"]):
            a.copy_(b)
        d.conv_cons_to_prim(ng, *cur, u, P, stream=raw)
        for _ in range(st["case"]["steps"]):
            dt = CFL * d.time_step(ng, cur[0], u, P, stream=raw)
            if not d.minimum_internal_energy(*cur, stream=raw) >= 0.0:
                raise RuntimeError("negative internal energy")
            d.hydro_reconstruction(1, dt / 2, cur[0], u, P, None, *rec, None, stream=raw)
            d.godunov_scheme(0, dt, *cur, None, *rec, None, *new, None, stream=raw)
            d.boundary_conditions(*new, stream=raw)
            cur, new = new, cur
            d.conv_cons_to_prim(ng, *cur, u, P, stream=raw)
    torch.cuda.current_stream().wait_stream(s)
    return list(cur) + [u, P]


def _run_adjoint(st):
    c, d = st["case"], st["handle"]
    rho, rhou, E, _ = st["init"]
    d.set_state(rho, rhou, E, device=True)
    d.adjoint_forward(c["steps"], cfl=CFL, checkpoint_every=c["every"], precision=c["precision"])
    out = d.get_state(out=tuple(st["out"]), device=True)
    d.adjoint_backward(st["lam"], st["grad"], device=True)
    return list(out) + [st["grad"]]


def _run_ensemble(st):
    c, e = st["case"], st["handle"]
    for d, init in zip(e.domains, st["init"]):
        d.set_state(*init, device=True)
    e.run(c["steps"], cfl=CFL, checkpoint_every=c["every"], adjoint_precision=c["precision"])
    out = [t for d, o in zip(e.domains, st["out"]) for t in d.get_state(out=o, device=True)]
    return out + e.adjoint(st["lam"], st["grad"], device=True)


# ---- the same outputs in plain torch, 64 bits -------------------------------------
def _at(a, d, s):
    """Value of the cell at offset s along d (the wrapped ends are ghost cells)."""
    return torch.roll(a, -s, dims=2 - d)


class _Step:
    """One MUSCL-Hancock step on full arrays with ghosts."""

    def __init__(self, case, mesh):
        self.c, self.m, self.nd = case, mesh, mesh.nd
        self.gm1 = case["gamma"] - 1
        nd = self.nd
        self.half = [(self.m.dx[d] + _at(self.m.dx[d], d, 1)) / 2 for d in range(nd)]

    def limited(self, R, L):
        ok = R * L > 0
        one = torch.ones_like(R)
        r, l = torch.where(ok, R, one), torch.where(ok, L, one)
        if self.c["limiter"] == "VanLeer":
            s = 2 * r * l / (r + l)
        elif self.c["limiter"] == "Minmod":
            s = torch.where(r.abs() < l.abs(), r, l)
        else:
            s = r * l * (r + l) / (r * r + l * l)
        return torch.where(ok, s, torch.zeros_like(s))

    def prim(self, q):
        nd = self.nd
        u = [q[1 + d] / q[0] for d in range(nd)]
        return [q[0]] + u + [self.gm1 * (q[1 + nd] - 0.5 * sum(q[1 + d] * u[d] for d in range(nd)))]

    def cons(self, w):
        nd = self.nd
        return [w[0]] + [w[0] * w[1 + d] for d in range(nd)] + [
            w[1 + nd] / self.gm1 + 0.5 * w[0] * sum(w[1 + d] * w[1 + d] for d in range(nd))]

    def flux(self, w, q, d):
        nd = self.nd
        f = [w[1 + d] * q[v] for v in range(nd + 2)]
        f[1 + d] = f[1 + d] + w[1 + nd]
        f[1 + nd] = f[1 + nd] + w[1 + nd] * w[1 + d]
        return f

    def sound(self, w):
        return torch.sqrt(self.c["gamma"] * w[1 + self.nd] / w[0])

    def riemann(self, qL, qR, d):
        nd, c = self.nd, self.c
        wL, wR = self.prim(qL), self.prim(qR)
        aL, aR = self.sound(wL), self.sound(wR)
        uL, uR, pL, pR = wL[1 + d], wR[1 + d], wL[1 + nd], wR[1 + nd]
        sL, sR = torch.minimum(uL - aL, uR - aR), torch.maximum(uL + aL, uR + aR)
        fL, fR = self.flux(wL, qL, d), self.flux(wR, qR, d)
        if c["riemann"] == "HLL":
            sL, sR = sL.clamp(max=0), sR.clamp(min=0)
            return [(sR * fL[v] - sL * fR[v] + sL * sR * (qR[v] - qL[v])) / (sR - sL) for v in range(nd + 2)]
        rL, rR = wL[0] * (sL - uL), wR[0] * (sR - uR)
        us = (pR - pL + rL * uL - rR * uR) / (rL - rR)
        ps = 0.5 * (pL + pR + rL * (us - uL) + rR * (us - uR))
        left, out = us > 0, sL * sR > 0
        S = torch.where(left, sL, sR)
        q = [torch.where(left, a, b) for a, b in zip(qL, qR)]
        w = [torch.where(left, a, b) for a, b in zip(wL, wR)]
        f = [torch.where(left, a, b) for a, b in zip(fL, fR)]
        un = w[1 + d]
        rs = q[0] * (S - un) / (S - us)
        Es = (S - un) / (S - us) * q[1 + nd] + (us - un) / (S - us) * (us * q[0] * (S - un) + w[1 + nd])
        star = [f[0] + S * (rs - q[0])] + [rs * us * w[1 + e] for e in range(nd)] + [f[1 + nd] + S * (Es - q[1 + nd])]
        star[1 + d] = rs * us * us + ps
        return [torch.where(out, a, b) for a, b in zip(f, star)]

    def gravity(self, rho):
        """Acceleration per dimension (a number or an array over x0)."""
        c, m = self.c, self.m
        if c["gravity"] == "Uniform":
            return _gvec(c)[: self.nd]
        dv = m.dv.expand(m.shape)[:, NG:-NG][NG:-NG]
        shell = (rho[NG:-NG, NG:-NG] * dv).sum((0, 1)) / dv.sum((0, 1))
        x, xc = m.x[0].reshape(-1), m.xc[0].reshape(-1)
        vol = 4 * math.pi / 3
        inside = torch.zeros_like(xc)
        inside[NG:] = vol * (xc[NG:] ** 3 - x[NG:-1] ** 3) * shell[NG:]
        inside[NG + 1:] += vol * (x[NG + 1:-1] ** 3 - xc[NG:-1] ** 3) * shell[NG:-1]
        M = c["central_mass"] + torch.cumsum(inside, 0)
        return [(-G_NEWTON * M / xc ** 2).view(1, 1, -1), 0.0, 0.0][: self.nd]

    def source(self, d, k, wL, wR):
        """Geometric terms of dimension d on a spherical grid, k = dt / dv."""
        nd, m = self.nd, self.m
        out = [0.0] * (nd + 2)
        if not m.spherical or d == 2:
            return out
        a, b = m.ds[d]
        kd = k * (b - a)
        out[1 + d] = out[1 + d] + kd * (wL[1 + nd] + wR[1 + nd]) / 2
        if d == 0:
            for e in (2, 3):
                out[1] = out[1] + kd * (wL[0] * wL[e] ** 2 + wR[0] * wR[e] ** 2) / 4
                out[e] = out[e] - k * m.rfac * (wR[0] * wR[e] * wR[1] * b + wL[0] * wL[e] * wL[1] * a)
        else:
            out[2] = out[2] + kd * m.cot * (wL[0] * wL[3] ** 2 + wR[0] * wR[3] ** 2) / 4
            out[3] = out[3] - k * m.pfac * (wR[0] * wR[3] * wR[2] * b + wL[0] * wL[3] * wL[2] * a)
        return out

    def dt(self, q):
        w = self.prim(q)
        a = self.sound(w)
        return CFL / float(sum((w[1 + d].abs() + a) / self.m.width[d] for d in range(self.nd)).max())

    def __call__(self, q, dt):
        nd, m = self.nd, self.m
        hydro, fx = q[: nd + 2], q[nd + 2:]
        w = self.prim(hydro)
        g = self.gravity(q[0])

        def faces(v, d):
            up, down = _at(v, d, 1) - v, v - _at(v, d, -1)
            s = self.limited(up / self.half[d], down / _at(self.half[d], d, -1)) * (m.dx[d] / 2)
            return v - s, v + s

        pr, qc, mass = [], [], []
        for d in range(nd):
            lo, hi = zip(*(faces(v, d) for v in w))
            pr.append((lo, hi))
            qc.append([self.cons(lo), self.cons(hi)])
        rho0 = [[qc[d][s][0] for s in (0, 1)] for d in range(nd)]
        mom0 = [[qc[d][s][1:1 + nd] for s in (0, 1)] for d in range(nd)]
        k = dt / 2 / m.dv
        inc = [0.0] * (nd + 2)
        for d in range(nd):
            fL, fR = (self.flux(pr[d][s], qc[d][s], d) for s in (0, 1))
            mass.append((fL[0], fR[0]))
            src = self.source(d, k, *pr[d])
            inc = [inc[v] + k * (fL[v] * m.ds[d][0] - fR[v] * m.ds[d][1]) + src[v] for v in range(nd + 2)]
        for d in range(nd):
            for s in (0, 1):
                new = [a + b for a, b in zip(qc[d][s], inc)]
                for e in range(nd):
                    new[1 + e] = new[1 + e] + dt / 2 * g[e] * rho0[d][s]
                    new[1 + nd] = new[1 + nd] + dt / 2 * g[e] * mom0[d][s][e]
                qc[d][s] = new
        del pr, w
        xf = []
        for x in fx:
            fc = [faces(x, d) for d in range(nd)]
            xi = sum(k * (fc[d][0] * mass[d][0] * m.ds[d][0] - fc[d][1] * mass[d][1] * m.ds[d][1]) for d in range(nd))
            xf.append([[(fc[d][s] * rho0[d][s] + xi) / qc[d][s][0] for s in (0, 1)] for d in range(nd)])
        del rho0, mom0, mass
        k = dt / m.dv
        out, xn = list(hydro), [x * q[0] for x in fx]
        for d in range(nd):
            F = self.riemann([_at(v, d, -1) for v in qc[d][1]], qc[d][0], d)
            src = self.source(d, k, *(self.prim(qc[d][s]) for s in (0, 1))) if m.spherical else [0.0] * (nd + 2)
            for v in range(nd + 2):
                out[v] = out[v] + k * (F[v] * m.ds[d][0] - _at(F[v], d, 1) * m.ds[d][1]) + src[v]
            out[1 + d] = out[1 + d] + dt * g[d] * hydro[0]
            out[1 + nd] = out[1 + nd] + dt * g[d] * hydro[1 + d]
            for f in range(len(fx)):
                X = torch.where(F[0] < 0, xf[f][d][0], _at(xf[f][d][1], d, -1)) * F[0]
                xn[f] = xn[f] + k * (X * m.ds[d][0] - _at(X, d, 1) * m.ds[d][1])
        return m.fill(out + [(x / out[0]).clamp(0, 1) for x in xn])


def _gradient(step, states, dts, lam):
    """dJ/dU^0 (interior) from dJ/dU^N, step by step backwards."""
    nd = step.nd
    for q, dt in zip(reversed(states), reversed(dts)):
        q = [t.detach().requires_grad_(True) for t in q]
        with torch.enable_grad():
            new = step(step.m.fill(q), dt)
        grads = torch.autograd.grad(new, q, [lam[v] for v in range(nd + 2)])
        lam = torch.zeros_like(lam)
        for v in range(nd + 2):
            lam[(v,) + step.m.inner] = grads[v][step.m.inner]
    return lam


def _exact_run(case, seed, dev, keep=False):
    mesh = _Mesh(case, dev)
    step = _Step(case, mesh)
    q = _initial(case, mesh, seed)
    states, dts, t, n = [], [], 0.0, 0
    while (n < case["steps"]) if case["steps"] else (t < 0.2):
        dt = step.dt(q)
        if not case["steps"]:
            dt = min(dt, 0.2 - t)
        if keep:
            states.append(q)
            dts.append(dt)
        q = step(q, dt)
        n += 1
        t = 0.2 if not case["steps"] and dt == 0.2 - t else t + dt
    return step, q, states, dts


@functools.lru_cache(maxsize=1)
def _device():
    return torch.device("cuda", 0) if torch.cuda.is_available() else torch.device("cpu")


@torch.no_grad()
def exact(case, seed):
    dev, nd = _device(), case["ndim"]
    if case["kind"] == "ensemble":
        outs, grads = [], []
        for p, m in enumerate(_problems(case)):
            step, q, states, dts = _exact_run(m, 1000 * seed + p, dev, keep=True)
            outs += list(_split(q, 2)[:3])
            grads.append(_gradient(step, states, dts, _energy_adjoint(step.m)))
        return outs + grads
    step, q, states, dts = _exact_run(case, seed, dev, keep=case["kind"] == "adjoint")
    rho, rhou, E, fx = _split(q, nd)
    out = [rho, rhou, E] + ([] if fx is None else [fx])
    if case["kind"] == "stages":
        w = step.prim(q)
        out += [torch.stack(w[1:1 + nd]), w[1 + nd]]
    if case["kind"] == "adjoint":
        out.append(_gradient(step, states, dts, _objective_adjoint(case, step.m, seed)))
    return out
