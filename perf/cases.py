"""The solves this framework is used for, as timed and checked cases.

Every case goes through the public entry points: `Solver.step` (one solve),
`Solver.diagnostics` (the history a run records) and `Batch.step` (many solves in one
CUDA graph).  Families (the `family` of a case):

  tgv        3D Taylor-Green vortex, Navier-Stokes, on a periodic box: the headline
             solve (supersonic, KEEP/SLAU hybrid) and the plain low-Mach SLAU one, FP64
             and mixed, Central-6 and ME4 viscous stencils, with the run's history
             (diagnostics) where `history` is set
  etgv       3D inviscid Taylor-Green vortex, KEEP, RK4
  channel    3D Navier-Stokes shear layer between no-slip walls in y (KEEP-6, Central-6)
  les        3D large-eddy simulation of decaying turbulence (SLAU-6, selective
             mixed-scale model), one solve
  les_batch  a serving mix: several of those, of uneven sizes, in one batched step
  vortex     one 2D isentropic-vortex convection (KEEP, RK4)
  ensemble   many of those, of uneven sizes, in one batched step
  tube       2D inviscid shock tube between non-periodic x ends (SLAU-6, TVD hybrid)

The initial fields are developed ones (seeded modes with a compressive part and
pressure and density variations on top of the analytic vortex), so that the hybrid
scheme meets shock-capturing faces, as a run past its first steps does.
"""
import math

import numpy as np
import torch

GAMMA, R_GAS, PR, PRT, THRESHOLD = 1.4, 287.03, 0.71, 0.9, 0.4
EXACT_CELLS = 20_000_000  # largest interior for which `exact` is computed

VORTEX_SIDES = (64, 96, 128, 192, 256, 384, 512)
LES_SIDES = (32, 48, 64, 96, 128)


def listed():
    return [
        # the reference's own shock-tube test: 513 x 7 nodes, thousands of tiny steps
        dict(name="tube_513x7_slau6", family="tube", nx=513, ny=7, steps=10, precision="fp64"),
        # the Euler-vortex convergence study at its default size
        dict(name="vortex_252_keep6", family="vortex", n=252, order=6, steps=10, precision="fp64"),
        # a 60^3 inviscid Taylor-Green run (20 000 such steps in the reference's test)
        dict(name="etgv_60_keep6", family="etgv", nx=60, ny=60, nz=60, order=6, steps=1, precision="fp64"),
        # the plain method: 64^3, SLAU-6, Mach 0.1, with the history every few steps
        dict(name="tgv_64_slau6_history", family="tgv", nx=64, ny=64, nz=64, scheme="SLAU", stencil="Central",
             mach=0.1, steps=4, history=True, precision="fp64"),
        # one LES request alone, an odd size
        dict(name="les_81_slau6_mixed", family="les", n=81, steps=1, precision="mixed"),
        # a walled box of ragged sides
        dict(name="channel_190x125x95_keep6", family="channel", nx=190, ny=125, nz=95, steps=1, precision="fp64"),
        # a ragged supersonic box with the ME4 viscous stencil
        dict(name="tgv_161x143x117_hybrid6_me4", family="tgv", nx=161, ny=143, nz=117, scheme="Hybrid",
             stencil="ME4Base", mach=1.25, steps=1, history=False, precision="fp64"),
        # the batched 2D ensemble, both forms
        dict(name="ensemble_64_keep4", family="ensemble", count=64, draw_seed=0, steps=1, precision="fp64"),
        dict(name="ensemble_64_keep4_mixed", family="ensemble", count=64, draw_seed=0, steps=1, precision="mixed"),
        # the serving mix: one resident request of every size
        dict(name="les_mix_slau6_mixed", family="les_batch", sides="32,48,64,96,128", steps=1, precision="mixed"),
        # the supersonic vortex at 256^3 in the mixed form
        dict(name="tgv_256_hybrid6_mixed", family="tgv", nx=256, ny=256, nz=256, scheme="Hybrid", stencil="Central",
             mach=1.25, steps=1, history=False, precision="mixed"),
        # the large single solve
        dict(name="tgv_512_hybrid6_me4", family="tgv", nx=512, ny=512, nz=512, scheme="Hybrid", stencil="ME4Base",
             mach=1.25, steps=1, history=False, precision="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed families and ranges (odd sizes included)."""
    family = rng.choice(["tgv", "tgv", "tgv", "etgv", "channel", "les", "les_batch", "vortex", "ensemble", "tube"])
    precision = rng.choice(["fp64", "mixed"])
    if family == "tgv":
        n = _log(rng, 32, 320)
        scheme = rng.choice(["Hybrid", "Hybrid", "SLAU", "KEEP"])
        return dict(family="tgv", nx=n, ny=max(8, int(n * rng.uniform(0.5, 1.0))),
                    nz=max(8, int(n * rng.uniform(0.5, 1.0))), scheme=scheme,
                    stencil=rng.choice(["Central", "ME4Base"]), mach=0.1 if scheme == "SLAU" else 1.25,
                    steps=rng.choice([1, 2, 3]), history=rng.random() < 0.3, precision=precision)
    if family == "etgv":
        n = _log(rng, 24, 200)
        return dict(family="etgv", nx=n, ny=max(8, int(n * rng.uniform(0.6, 1.0))),
                    nz=max(8, int(n * rng.uniform(0.6, 1.0))), order=rng.choice([2, 4, 6]), steps=rng.choice([1, 2]),
                    precision=precision)
    if family == "channel":
        n = _log(rng, 32, 240)
        return dict(family="channel", nx=n, ny=max(12, int(n * rng.uniform(0.4, 1.0))),
                    nz=max(12, int(n * rng.uniform(0.4, 1.0))), steps=1, precision="fp64")
    if family == "les":
        return dict(family="les", n=_log(rng, 32, 160), steps=rng.choice([1, 2]), precision=precision)
    if family == "les_batch":
        sides = [rng.choice(LES_SIDES) for _ in range(rng.randint(2, 6))]
        return dict(family="les_batch", sides=",".join(str(s) for s in sides), steps=1, precision="mixed")
    if family == "vortex":
        return dict(family="vortex", n=_log(rng, 48, 700), order=rng.choice([4, 6]), steps=rng.choice([1, 5, 10]),
                    precision=precision)
    if family == "ensemble":
        return dict(family="ensemble", count=rng.randint(8, 64), draw_seed=rng.randint(1, 10 ** 6), steps=1,
                    precision=precision)
    return dict(family="tube", nx=_log(rng, 200, 2000), ny=rng.choice([7, 9, 33, 64, 129]), steps=rng.choice([2, 10]),
                precision="fp64")


# ------------------------------------------------------------------ physics and grids --
def _members(case):
    """(n, beta, mach) of a batched ensemble's vortices."""
    rng = np.random.default_rng(case["draw_seed"])
    return [(int(rng.choice(VORTEX_SIDES)), float(rng.uniform(1.0, 5.0)), float(rng.uniform(0.1, 0.8)))
            for _ in range(case["count"])]


def _sides(case):
    return [int(s) for s in case["sides"].split(",")]


def _solves(case):
    """The solves of a case, each a dict of plain values: interior extents (x, y, z; a
    non-periodic axis counts its cells between the two boundary cells), scheme, constants,
    spacings and dt."""
    f = case["family"]
    base = dict(family=f, gamma=GAMMA, R=R_GAS, Pr=PR, Prt=PRT, threshold=THRESHOLD, visc="Euler", stencil="Central",
                tvd="hybrid", rk=3, walls="", order=6, scheme="KEEP", les=False)
    out = []
    if f == "tgv":
        # NSTGV's dimensional set-up: T = 294.4 K, L0 = 1.524 mm, Re = 1600, box 2 pi L0
        T0, L0, Re, mach = 530.0 * 5.0 / 9.0, 1.524e-3, 1600.0, case["mach"]
        c0 = math.sqrt(GAMMA * R_GAS * T0)
        V0 = mach * c0
        rho0 = _sutherland(T0) * Re / (V0 * L0)
        h = [2.0 * math.pi * L0 / n for n in (case["nx"], case["ny"], case["nz"])]
        out.append(dict(base, n=(case["nx"], case["ny"], case["nz"]), h=h, dt=0.35 * min(h) / (V0 + c0),
                        scheme=case["scheme"], stencil=case["stencil"], visc="NS", V0=V0, rho0=rho0,
                        p0=rho0 * R_GAS * T0, mach=mach))
    elif f == "etgv":
        h = [2.0 * math.pi / n for n in (case["nx"], case["ny"], case["nz"])]
        out.append(dict(base, n=(case["nx"], case["ny"], case["nz"]), h=h, dt=0.35 * min(h) / 1.6, order=case["order"],
                        rk=4, V0=0.4, rho0=1.0, p0=1.0 / GAMMA, mach=0.4))
    elif f == "channel":
        T0, L, mach = 300.0, 2.0e-3, 0.4
        c0 = math.sqrt(GAMMA * R_GAS * T0)
        V0 = mach * c0
        rho0 = _sutherland(T0) * 800.0 / (V0 * L)
        h = [L / n for n in (case["nx"], case["ny"], case["nz"])]
        out.append(dict(base, n=(case["nx"], case["ny"], case["nz"]), h=h, dt=0.2 * min(h) / (V0 + c0), visc="NS",
                        walls="y", V0=V0, rho0=rho0, p0=rho0 * R_GAS * T0, mach=mach))
    elif f in ("les", "les_batch"):
        for n in ([case["n"]] if f == "les" else _sides(case)):
            T0, L0, mach = 300.0, 1.0e-3, 0.3
            c0 = math.sqrt(GAMMA * R_GAS * T0)
            V0 = mach * c0
            rho0 = _sutherland(T0) * 800.0 / (V0 * L0)
            h = [2.0 * math.pi * L0 / n] * 3
            out.append(dict(base, n=(n, n, n), h=h, dt=0.3 * h[0] / (V0 + c0), scheme="SLAU", visc="LES", les=True,
                            V0=V0, rho0=rho0, p0=rho0 * R_GAS * T0, mach=mach))
    elif f in ("vortex", "ensemble"):
        members = [(case["n"], 4.0, 0.4)] if f == "vortex" else _members(case)
        for n, beta, mach in members:
            h = [10.0 / n] * 2
            out.append(dict(base, n=(n, n), h=h, dt=0.4 * h[0] / (1.0 + mach), order=case.get("order", 4), rk=4, R=1.0,
                            beta=beta, mach=mach))
    elif f == "tube":
        nx, ny = case["nx"] - 2, case["ny"] - 6
        h = [1.0 / (nx + 1), 0.1 / (ny + 5)]
        out.append(dict(base, n=(nx, ny), h=h, dt=0.1 * min(h), scheme="SLAU", walls="x", R=1.0))
    else:
        raise ValueError(f"unknown family {f!r}")
    return out


def _sutherland(T):
    return 1.716e-5 * (273.2 + 111.0) / (T + 111.0) * (T / 273.2) ** 1.5


def _ghosts(s):
    return [1 if "xyz"[a] in s["walls"] else s["order"] // 2 for a in range(len(s["n"]))]


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _field(s, seed, dev):
    """Q / J of a solve on its padded grid, ghost cells not yet filled: a tensor
    (nv, nz, ny, nx), or (nv, ny, nx) in 2D, x fastest."""
    dim = len(s["n"])
    g = _ghosts(s)
    rng = np.random.default_rng([seed, 7919])
    ax = []
    for a in range(dim):
        c = (torch.arange(s["n"][a] + 2 * g[a], device=dev, dtype=torch.float64) - g[a] + 0.5) * s["h"][a]
        ax.append(c.reshape([-1 if d == dim - 1 - a else 1 for d in range(dim)]))
    gam = s["gamma"]
    f = s["family"]
    one = torch.ones([s["n"][a] + 2 * g[a] for a in reversed(range(dim))], device=dev, dtype=torch.float64)
    if f == "tube":
        left = (ax[0] < 0.5 + 0.02 * float(rng.uniform(-1, 1))).to(torch.float64) * one
        bump = 1.0 + 0.02 * torch.sin(9.0 * ax[0] + float(rng.uniform(0, 6))) * one
        rho, p, vel = (0.125 + 0.875 * left) * bump, (0.1 + 0.9 * left) * bump, [0.05 * left, 0.0 * one]
    elif dim == 2:
        L = 10.0
        x0, y0 = (float(v) for v in rng.uniform(0.3, 0.7, 2) * L)
        dx = torch.remainder(ax[0] - x0 + 0.5 * L, L) - 0.5 * L
        dy = torch.remainder(ax[1] - y0 + 0.5 * L, L) - 0.5 * L
        r2 = dx * dx + dy * dy
        e = torch.exp(0.5 * (1.0 - r2))
        b = s["beta"] * float(rng.uniform(0.9, 1.0))
        rho = (1.0 - (gam - 1.0) * b * b / (8.0 * gam * math.pi ** 2) * e * e) ** (1.0 / (gam - 1.0))
        p = rho ** gam / gam
        vel = [s["mach"] - b / (2.0 * math.pi) * dy * e, b / (2.0 * math.pi) * dx * e]
    else:
        X = [ax[a] * (2.0 * math.pi / (s["n"][a] * s["h"][a])) + float(rng.uniform(0, 6.0)) for a in range(3)]
        V0, rho0, p0, m2 = s["V0"], s["rho0"], s["p0"], gam * s["mach"] ** 2
        sx, cx, sy, cy, sz, cz = (t for a in range(3) for t in (torch.sin(X[a]), torch.cos(X[a])))
        if f in ("les", "les_batch"):
            vel = [0.0 * one, 0.0 * one, 0.0 * one]
            modes, solenoidal, compressive = 24, 0.12, 0.01
        elif f == "channel":
            eta = ax[1] / (s["n"][1] * s["h"][1])
            env = 4.0 * eta * (1.0 - eta)
            vel = [V0 * env * one, 0.0 * one, 0.0 * one]
            modes, solenoidal, compressive = 6, 0.03, 0.005
        else:
            vel = [V0 * sx * cy * cz, -V0 * cx * sy * cz, 0.0 * one]
            modes, solenoidal, compressive = 8, 0.05, 0.03
        pert = 0.0 * one
        for _ in range(modes):
            k = rng.integers(-4, 5, 3).astype(float)
            if not k.any():
                k[0] = 1.0
            ph = k[0] * X[0] + k[1] * X[1] + k[2] * X[2] + float(rng.uniform(0, 2 * math.pi))
            d = np.cross(k, rng.standard_normal(3))
            d = d / (np.linalg.norm(d) + 1e-12) * solenoidal + k / np.linalg.norm(k) * compressive
            w = torch.cos(ph)
            for a in range(3):
                vel[a] = vel[a] + (V0 * float(d[a])) * w
            pert = pert + 0.02 * torch.sin(ph)
            del ph, w
        if f == "channel":
            vel = [v * torch.clamp(env, min=0.0) if a else v for a, v in enumerate(vel)]
        p = p0 * (1.0 + m2 / 16.0 * (torch.cos(2 * X[0]) + torch.cos(2 * X[1])) * (torch.cos(2 * X[2]) + 2.0) * 0.5
                  + 0.3 * min(1.0, m2) * pert)
        rho = rho0 * (1.0 + 0.2 * min(1.0, m2) * pert) * one
        del pert
    vol = 1.0
    for h in s["h"]:
        vol *= h
    q = torch.empty([dim + 2] + list(one.shape), device=dev, dtype=torch.float64)
    q[0] = rho * vol
    ke = 0.0
    for a in range(dim):
        q[1 + a] = rho * vel[a] * vol
        ke = ke + vel[a] * vel[a]
    q[dim + 1] = (p / (gam - 1.0) + 0.5 * rho * ke) * vol
    return q


def _config(s, precision):
    from ouxsbli_b200.config import SolverConfig
    dim = len(s["n"])
    g = _ghosts(s)
    ext = [s["n"][a] + 2 * g[a] for a in range(dim)] + [1] * (3 - dim)
    d = [np.full(ext[a] - 1, s["h"][a]) for a in range(dim)] + [None] * (3 - dim)
    kw = {}
    if "x" in s["walls"]:
        kw["bc_x"] = 1
    if "y" in s["walls"]:
        kw["bc_y"] = 1
        kw["boundary"] = {"y_lo": "noslip_wall", "y_hi": "noslip_wall"}
    return SolverConfig(dim=dim, nx=ext[0], ny=ext[1], nz=ext[2], order=s["order"], scheme=s["scheme"], visc=s["visc"],
                        visc_stencil=s["stencil"], tvd=s["tvd"], slau="HRSLAU2", rk=s["rk"], precision=precision,
                        gamma=s["gamma"], R=s["R"], Pr=s["Pr"], Prt=s["Prt"], threshold=s["threshold"], dt=s["dt"],
                        dx=d[0], dy=d[1], dz=d[2], **kw)


def _view(solver):
    """The solve's state as the caller sees it: its variables (over the Jacobian) on the
    padded grid, (nv, nz, ny, nx) or (nv, ny, nx), a view of the state buffer."""
    c, lay = solver.cfg, solver.layout
    size, stride = [c.nv, c.ny, c.nx], [lay.var_stride, lay.row_stride, 1]
    if c.dim == 3:
        size.insert(1, c.nz)
        stride.insert(1, lay.plane_stride)
    q = torch.as_strided(solver.state, size, stride)
    return q


def _parts(q):
    return {"rho": q[0], "mom": q[1:-1], "E": q[-1]}


# --------------------------------------------------------------------------- the cases --
def prepare(case, seed):
    from ouxsbli_b200.solver import Solver
    solvers = []
    for i, s in enumerate(_solves(case)):
        q = _field(s, seed + 1000 * i, _device())
        dim = len(s["n"])
        # the reference's order QJ(nx, nv, ny, nz), x fastest
        host = q.movedim(0, dim - 1).contiguous().cpu().numpy()
        del q
        solver = Solver(_config(s, case["precision"]), "cuda:0")
        solver.set_state(host.transpose(tuple(reversed(range(dim + 1)))))
        solver.fill_ghosts()
        solvers.append(solver)
    state = {"case": case, "solvers": solvers, "views": [_view(s) for s in solvers], "batch": None}
    if case["family"] in ("ensemble", "les_batch"):
        from ouxsbli_b200.batch import Batch, Tuning
        state["batch"] = Batch(solvers, Tuning(mode="graph"))
    return state


def run(state):
    case = state["case"]
    if state["batch"] is not None:
        state["batch"].step(case["steps"])
        return _outputs(case, state["views"])
    solver = state["solvers"][0]
    solver.step(case["steps"])
    out = _parts(state["views"][0])
    if case.get("history"):
        out["history"] = np.array(solver.diagnostics())
    return out


def _outputs(case, q):
    """The states of a batch: density, momentum and energy apart where the variables'
    magnitudes differ; an ensemble's nondimensional states whole, one array a solve."""
    return q if case["family"] == "ensemble" else [_parts(v) for v in q]


# floating-point operations per cell and Runge-Kutta stage, counted from the formulas:
# one face per axis of a cell (each face value serves two cells), plus the cell's own terms
_CONV = {2: 40, 4: 120, 6: 230}
_SLAU6 = 5 * 30 + 130
_VISC = {"Central": 270, "ME4Base": 260}


def work(case):
    nbytes, flops = 0.0, 0.0
    for s in _solves(case):
        dim = len(s["n"])
        cells = float(np.prod(s["n"]))
        stages = 3 if s["rk"] == 3 else 4
        face = _SLAU6 if s["scheme"] == "SLAU" else _CONV[s["order"]]
        per = dim * face * (1.0 if dim == 3 else 0.8) + 20 + 9 * (dim + 2)
        if s["visc"] != "Euler":
            per += dim * _VISC[s["stencil"]] + 9 * 9 + 15
        if s["scheme"] != "KEEP":
            per += 40
        if s["les"]:
            per += dim * 120 + 450
        nbytes += 2.0 * 8.0 * (dim + 2) * cells
        flops += per * cells * stages * case["steps"]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # measured against `exact` over the families, sizes 30 to 600 a side and up to ten
    # steps: FP64 1.0e-15 (the momentum of the Mach 0.1 solves), mixed 8.5e-8 where no
    # face changes its discrete decision, and 7.4e-7 where one does (SLAU's pressure
    # wiggle detector and TVD switch read differences that FP32 fields hold to few digits)
    if case["precision"] != "mixed":
        return {"rel": 4e-15}
    if case["family"].startswith("les") or case.get("scheme") == "SLAU":
        return {"rel": 3e-6}
    return {"rel": 1e-6} if case.get("scheme") == "Hybrid" else {"rel": 4e-7}


# ------------------------------------------------------------------------------- exact --
class _Exact:
    """One solve in plain torch, 64 bits: the finite-volume scheme written from its
    formulas on whole padded arrays (uniform spacings)."""

    def __init__(self, s, q):
        self.s, self.q = s, q
        self.dim = len(s["n"])
        self.g = _ghosts(s)
        self.ng = s["order"] // 2
        self.vol = float(np.prod(s["h"]))
        self.J = 1.0 / self.vol

    # array axis of grid axis a, and a slice of it
    def ax(self, v, a):
        return v.dim() - 1 - a

    def cut(self, v, a, lo, n):
        return v.narrow(self.ax(v, a), lo, n)

    def wall(self, a):
        return "xyz"[a] in self.s["walls"]

    def fill(self, q):
        for a in range(self.dim):
            if self.wall(a):
                continue
            g, n = self.g[a], self.s["n"][a]
            i = torch.remainder(torch.arange(n + 2 * g, device=q.device) - g, n) + g
            q.copy_(q.index_select(self.ax(q, a), i))
        for a in range(self.dim):
            if not self.wall(a):
                continue
            n = self.s["n"][a] + 2
            for b, src in ((0, 1), (n - 1, n - 2)):
                v = self.cut(q, a, src, 1).clone()
                if a == 1:  # no-slip wall: the neighbour's density and pressure
                    ke = sum(v[1 + c] * v[1 + c] for c in range(self.dim))
                    v[self.dim + 1] = v[self.dim + 1] - 0.5 * ke / v[0]
                    v[1:self.dim + 1] = 0.0
                self.cut(q, a, b, 1).copy_(v)

    def prim(self, q):
        s, W = self.s, {}
        over = 1.0 / q[0]
        W["r"] = self.J * q[0]
        W["v"] = [q[1 + a] * over for a in range(self.dim)]
        ke = sum(v * v for v in W["v"])
        W["p"] = (s["gamma"] - 1.0) * (self.J * q[self.dim + 1] - 0.5 * W["r"] * ke)
        W["T"] = W["p"] / (s["R"] * W["r"])
        if s["visc"] != "Euler":
            W["mu"] = 1.716e-5 * 384.2 * 273.2 ** -1.5 / (W["T"] + 111.0) * (W["T"] * torch.sqrt(W["T"]))
        if s["scheme"] != "KEEP":
            W["sen"] = self.sensor(W["v"])
        if s["visc"] != "Euler":
            W["D"] = [[self.node(W["v"][c], a) for a in range(3)] for c in range(3)]
        if s["les"]:
            W["mut"], W["qc"] = self.sgs(W)
        return W

    def shift(self, v, a, o):
        return torch.roll(v, -o, self.ax(v, a))

    def node(self, f, a):
        S = lambda o: self.shift(f, a, o)  # noqa: E731
        if self.s["stencil"] == "ME4Base":
            d = 2.0 / 3.0 * (S(1) - S(-1)) - (S(2) - S(-2)) / 12.0
        else:
            d = (S(3) - S(-3)) / 60.0 - 0.15 * (S(2) - S(-2)) + 0.75 * (S(1) - S(-1))
        return d / self.s["h"][a]

    def sensor(self, v):
        d = [[(self.shift(v[c], a, 1) - self.shift(v[c], a, -1)) * (0.5 / self.s["h"][a]) for a in range(self.dim)]
             for c in range(self.dim)]
        div = sum(d[a][a] for a in range(self.dim))
        if self.dim == 3:
            rot = (d[2][1] - d[1][2]) ** 2 + (d[0][2] - d[2][0]) ** 2 + (d[1][0] - d[0][1]) ** 2
        else:
            rot = (d[1][0] - d[0][1]) ** 2
        f = torch.clamp(div * div / (div * div + rot + 1e-12), max=1.0)
        for a in range(self.dim):  # the outermost cells copy their neighbour
            n = f.shape[self.ax(f, a)]
            self.cut(f, a, 0, 1).copy_(self.cut(f, a, 1, 1).clone())
            self.cut(f, a, n - 1, 1).copy_(self.cut(f, a, n - 2, 1).clone())
        return f

    def sgs(self, W):
        """Selective mixed-scale viscosity and the test-filtered kinetic energy."""
        h = self.s["h"]
        v = W["v"]
        vt = [c + 0.25 * sum(self.shift(c, a, 1) - 2.0 * c + self.shift(c, a, -1) for a in range(3)) for c in v]
        # cells next to the outermost layer are not filtered (their whole neighbourhood)
        inner = torch.zeros_like(v[0], dtype=torch.bool)
        inner[2:-2, 2:-2, 2:-2] = True
        qc = sum((a - b) ** 2 for a, b in zip(v, vt)) * 0.5

        def vort(u):
            d = lambda c, a: (self.shift(u[c], a, 1) - self.shift(u[c], a, -1)) * (0.5 / h[a])  # noqa: E731
            return [d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)]

        o, t = vort(v), vort(vt)
        qc = torch.where(inner, qc, torch.zeros_like(qc))
        t = [torch.where(inner, b, a) for a, b in zip(o, t)]
        o2, t2 = sum(a * a for a in o), sum(a * a for a in t)
        d2 = sum((a - b) ** 2 for a, b in zip(o, t))
        cross = 2.0 * torch.sqrt(o2) * torch.sqrt(t2)
        den = cross + t2 + o2 - d2
        tan2 = torch.where(den.abs() < 1e-30, torch.zeros_like(den), (cross - t2 - o2 + d2) / den)
        f = torch.clamp((tan2 / math.tan(math.pi / 18.0) ** 2) ** 2, max=1.0)
        d = lambda c, a: (self.shift(v[c], a, 1) - self.shift(v[c], a, -1)) * (0.5 / h[a])  # noqa: E731
        S2 = 2.0 * sum(d(a, a) ** 2 for a in range(3))
        S2 = S2 + (d(1, 0) + d(0, 1)) ** 2 + (d(2, 1) + d(1, 2)) ** 2 + (d(0, 2) + d(2, 0)) ** 2
        inv = [1.0 / x for x in h]
        l1, l2 = math.log(min(inv) / inv[0]), math.log(min(inv) / inv[1])
        delta = math.cosh(math.sqrt(4.0 * (l1 * l1 - l1 * l2 + l2 * l2) / 27.0)) * (inv[0] * inv[1] * inv[2]) ** (-1 / 3)
        mut = W["r"] * (f * 0.06 * S2 ** 0.25 * qc ** 0.25 * delta ** 1.5)
        for z in (mut, qc):  # the outer layer takes its image at distance n - 2
            for a in range(3):
                n = z.shape[self.ax(z, a)]
                self.cut(z, a, 0, 1).copy_(self.cut(z, a, n - 2, 1).clone())
                self.cut(z, a, n - 1, 1).copy_(self.cut(z, a, 1, 1).clone())
        return mut, qc

    # values of cells (face's left cell + off) for every face of the sweep along `a`
    def at(self, v, a, off):
        for b in range(self.dim):
            if b != a:
                v = self.cut(v, b, self.g[b], self.s["n"][b])
        lo, n = self.g[a] - 1 + off, self.s["n"][a] + 1
        size = v.shape[self.ax(v, a)]
        if lo >= 0 and lo + n <= size:
            return self.cut(v, a, lo, n)
        i = torch.clamp(torch.arange(lo, lo + n, device=v.device), 0, size - 1)  # never used where clamped
        return v.index_select(self.ax(v, a), i)

    def keep(self, W, a, order):
        m = order // 2
        pts = range(-m + 1, m + 1)
        C = lambda v: {o: self.at(v, a, o) for o in pts}  # noqa: E731
        r, p, T = C(W["r"]), C(W["p"]), C(W["T"])
        v = [C(c) for c in W["v"]]
        un = v[a]
        # pair weights by distance l = 1..m: central coefficients a_l, pairs (i, i + l) that straddle the face
        al = {2: [0.5], 4: [2.0 / 3.0, -1.0 / 12.0], 6: [0.75, -0.15, 1.0 / 60.0]}[order]
        F = [0.0] * (self.dim + 2)
        Rg = self.s["R"] / (self.s["gamma"] - 1.0)
        for l in range(1, m + 1):
            w = 2.0 * al[l - 1]
            for i in range(1 - l, 1):
                j = i + l
                c = w * 0.25 * (r[i] + r[j]) * (un[i] + un[j])
                F[0] = F[0] + c
                for d in range(self.dim):
                    F[1 + d] = F[1 + d] + c * 0.5 * (v[d][i] + v[d][j])
                F[1 + a] = F[1 + a] + w * 0.5 * (p[i] + p[j])
                e = c * 0.5 * (T[i] + T[j]) * Rg + c * 0.5 * sum(v[d][i] * v[d][j] for d in range(self.dim))
                F[-1] = F[-1] + e + w * 0.5 * (un[i] * p[j] + un[j] * p[i])
        return F

    def recon(self, v, a, order, plain):
        x = lambda o: self.at(v, a, o)  # noqa: E731
        if order == 2:
            return x(0), x(1)
        if order == 4:
            d = [x(o + 1) - x(o) for o in (-1, 0, 1)]
            b = (3.0 - 1.0 / 3.0) / (1.0 - 1.0 / 3.0)
            mm = self.minmod
            L = torch.where(plain, 0.5 * (d[0] + 2.0 * d[1]) / 3.0,
                            0.5 * (mm(d[0], b * d[1]) + 2.0 * mm(d[1], b * d[0])) / 3.0)
            Rr = torch.where(plain, 0.5 * (d[2] + 2.0 * d[1]) / 3.0,
                             0.5 * (mm(d[2], b * d[1]) + 2.0 * mm(d[1], b * d[2])) / 3.0)
            return x(0) + L, x(1) - Rr
        d = [x(o + 1) - x(o) for o in (-2, -1, 0, 1, 2)]
        pl = (-0.4 * d[0] + 2.2 * d[1] + 4.8 * d[2] - 0.6 * d[3]) / 12.0
        pr = (-0.6 * d[1] + 4.8 * d[2] + 2.2 * d[3] - 0.4 * d[4]) / 12.0
        mm = self.minmod

        def d33(p, q, r):
            return mm(p, 2 * q, 2 * r) - 2.0 * mm(q, 2 * p, 2 * r) + mm(r, 2 * p, 2 * q)

        dm = d[2] - d33(d[1], d[2], d[3]) / 6.0
        dl = d[1] - d33(d[0], d[1], d[2]) / 6.0
        dh = d[3] - d33(d[2], d[3], d[4]) / 6.0
        tl = (mm(dl, 4.0 * dm) + 2.0 * mm(dm, 4.0 * dl)) / 6.0
        tr = (mm(dh, 4.0 * dm) + 2.0 * mm(dm, 4.0 * dh)) / 6.0
        return x(0) + torch.where(plain, pl, tl), x(1) - torch.where(plain, pr, tr)

    @staticmethod
    def minmod(x, *others):
        s = torch.where(torch.signbit(x), -1.0, 1.0).to(x.dtype)
        m = x.abs()
        for y in others:
            m = torch.minimum(m, s * y)
        return s * torch.clamp(m, min=0.0)

    def slau(self, W, a, order, fd, wiggle):
        s = self.s
        plain = fd < s["threshold"]
        r1, r2 = self.recon(W["r"], a, order, plain)
        V = [self.recon(c, a, order, plain) for c in W["v"]]
        p1, p2 = self.recon(W["p"], a, order, plain)
        if wiggle and order > 2:
            x = [self.at(W["p"], a, o) for o in (-1, 0, 1, 2)]
            f = torch.minimum((x[1] - x[0]) * (x[2] - x[1]), (x[3] - x[2]) * (x[2] - x[1]))
            HR = torch.where(torch.signbit(f), 1.0, 0.0).to(f.dtype)
        else:
            HR = 1.0
        u1, u2 = V[a]
        c = 0.5 * (torch.sqrt(s["gamma"] * p1 / r1) + torch.sqrt(s["gamma"] * p2 / r2))
        Mp, Mm = u1 / c, u2 / c
        g = -torch.clamp(Mp, -1.0, 0.0) * torch.clamp(Mm, 0.0, 1.0)
        gv = (1.0 - g) * (r1 * u1.abs() + r2 * u2.abs()) / (r1 + r2)
        bp = torch.where(Mp.abs() < 1.0, 0.25 * (2.0 - Mp) * (Mp + 1.0) ** 2, (Mp > 0).to(Mp.dtype))
        bm = torch.where(Mm.abs() < 1.0, 0.25 * (2.0 + Mm) * (Mm - 1.0) ** 2, (Mm < 0).to(Mp.dtype))
        k1, k2 = 0.5 * sum(v[0] ** 2 for v in V), 0.5 * sum(v[1] ** 2 for v in V)
        q = torch.sqrt(k1 + k2)
        x = (1.0 - torch.clamp(q / c, max=1.0)) ** 2
        mass = 0.25 * (r1 * (u1 + gv + g * u1.abs()) + r2 * (u2 - gv - g * u2.abs()) - x * (p2 - p1) / c)
        pres = 0.5 * (p1 + p2 - (bp - bm) * (p2 - p1) + HR * q * (bp + bm - 1.0) * 0.5 * (r1 + r2) * c)
        m1, m2 = mass + mass.abs(), mass - mass.abs()
        F = [m1 + m2] + [m1 * v[0] + m2 * v[1] for v in V]
        F[1 + a] = F[1 + a] + pres
        gg = s["gamma"] / (s["gamma"] - 1.0)
        return F + [m1 * (p1 * gg / r1 + k1) + m2 * (p2 * gg / r2 + k2)]

    def conv(self, W, a, order):
        sch = self.s["scheme"]
        if sch == "KEEP":
            return self.keep(W, a, order)
        fd = 0.5 * (self.at(W["sen"], a, 0) + self.at(W["sen"], a, 1))
        S = self.slau(W, a, order, fd, sch == "SLAU")
        if sch == "SLAU":
            return S
        K = self.keep(W, a, order)
        cap = fd > self.s["threshold"]
        return [torch.where(cap, x, y) for x, y in zip(S, K)]

    def c6(self, v, a, diff):
        x = [self.at(v, a, o) for o in (-2, -1, 0, 1, 2, 3)]
        if diff:
            return (-0.0046875 * x[0] + 0.065104167 * x[1] - 1.171875 * (x[2] - x[3]) - 0.065104167 * x[4]
                    + 0.0046875 * x[5]) / self.s["h"][a]
        return (3.0 * (x[0] + x[5]) - 25.0 * (x[1] + x[4]) + 150.0 * (x[2] + x[3])) / 256.0

    def visc(self, W, a):
        """Stress components (x, y, z) and energy term of every face along a."""
        s = self.s
        cp = s["gamma"] * s["R"] / (s["gamma"] - 1.0)
        oth = [b for b in range(3) if b != a]
        tau, work = [None] * 3, [None] * 3
        if s["stencil"] == "ME4Base":
            acc = {}
            for o, w in ((-1, -1.0 / 24.0), (0, 26.0 / 24.0), (1, -1.0 / 24.0)):
                X = lambda v: [self.at(v, a, o + d) for d in (-1, 0, 1, 2)]  # noqa: E731,B023
                ip = lambda x: (9.0 * (x[1] + x[2]) - x[0] - x[3]) / 16.0  # noqa: E731
                df = lambda x: (1.125 * (x[2] - x[1]) - (x[3] - x[0]) / 24.0) / s["h"][a]  # noqa: E731
                mu = ip(X(W["mu"]))
                t = {"k": cp / s["Pr"] * mu * df(X(W["T"]))}
                for c in range(3):
                    vc = X(W["v"][c])
                    if c == a:
                        st = 2.0 / 3.0 * mu * (2.0 * df(vc) - ip(X(W["D"][oth[0]][oth[0]])) - ip(X(W["D"][oth[1]][oth[1]])))
                    else:
                        st = mu * (df(vc) + ip(X(W["D"][a][c])))
                    t["t%d" % c], t["w%d" % c] = st, ip(vc) * st
                for key, val in t.items():
                    acc[key] = acc.get(key, 0.0) + w * val
            return [acc["t%d" % c] for c in range(3)], acc["w0"] + acc["w1"] + acc["w2"] + acc["k"]
        mu = self.c6(W["mu"], a, False)
        mt = 0.5 * (mu + self.c6(W["mut"], a, False)) if s["les"] else None
        e = cp / s["Pr"] * mu * self.c6(W["T"], a, True)
        for c in range(3):
            dv = self.c6(W["v"][c], a, True)
            if c == a:
                d = 2.0 / 3.0 * (2.0 * dv - sum(self.c6(W["D"][b][b], a, False) for b in oth))
            else:
                d = dv + self.c6(W["D"][a][c], a, False)
            work[c] = self.c6(W["v"][c], a, False) * (mu * d)
            tau[c] = (mt if s["les"] else mu) * d
        e = e + sum(work)
        if s["les"]:
            H = cp * W["T"] + 0.5 * sum(v * v for v in W["v"]) + W["qc"]
            e = e - self.c6(W["mut"], a, False) * self.c6(H, a, True) / s["Prt"]
        return tau, e

    def visc_low(self, W, a):
        """The 2nd-order viscous face next to a wall."""
        s, h = self.s, self.s["h"]
        cp = s["gamma"] * s["R"] / (s["gamma"] - 1.0)
        x0, x1 = lambda v: self.at(v, a, 0), lambda v: self.at(v, a, 1)  # noqa: E731
        mu = 0.5 * (x0(W["mu"]) + x1(W["mu"]))
        e = cp / s["Pr"] * mu * (x1(W["T"]) - x0(W["T"])) / h[a]

        def nb(v, b, o):
            return self.shift(v, b, o)

        D = [[None] * 3 for _ in range(3)]
        for b in range(3):
            if b == a:
                for c in range(3):
                    D[c][a] = mu * (x1(W["v"][c]) - x0(W["v"][c])) / h[a]
                continue
            m = {o: x0(nb(W["mu"], b, o)) + x1(nb(W["mu"], b, o)) for o in (-1, 0, 1)}
            m1, m2 = 0.25 * (m[-1] + m[0]), 0.25 * (m[0] + m[1])
            for c in (a, b):
                f = {o: x0(nb(W["v"][c], b, o)) + x1(nb(W["v"][c], b, o)) for o in (-1, 0, 1)}
                D[c][b] = 0.25 * (m1 * (f[0] - f[-1]) + m2 * (f[1] - f[0])) / h[b]
        tau = []
        for c in range(3):
            if c == a:
                o = [b for b in range(3) if b != a]
                tau.append(2.0 / 3.0 * (2.0 * D[a][a] - D[o[0]][o[0]] - D[o[1]][o[1]]))
            else:
                tau.append(D[a][c] + D[c][a])
            e = e + 0.5 * (x0(W["v"][c]) + x1(W["v"][c])) * tau[c]
        return tau, e

    def index(self, like, a, b, face):
        """Cell index along axis b of every face of the sweep along a (the left cell when b == a)."""
        n = self.s["n"][b] + (1 if face else 0)
        i = torch.arange(n, device=like.device) + self.g[b] - (1 if face else 0)
        return i.reshape([-1 if d == self.ax(like, b) else 1 for d in range(like.dim())])

    def flux(self, W, a):
        s, order = self.s, self.s["order"]
        F = self.conv(W, a, order)
        if self.wall(a):
            n = s["n"][a] + 2
            f = self.index(F[0], a, a, True)
            for lo in ([4, 2] if order == 6 else [2] if order == 4 else []):
                low = ~((f >= 2) & (f <= n - 4)) if lo == 4 or order == 4 and lo == 2 else ~((f >= 1) & (f <= n - 3))
                F = [torch.where(low, y, x) for x, y in zip(F, self.conv(W, a, lo))]
        if s["visc"] != "Euler":
            tau, e = self.visc(W, a)
            if s["walls"]:  # Central-6 guard: faces 2 .. n-4, transverse cells 3 .. n-4
                ok = torch.ones_like(e, dtype=torch.bool)
                for b in range(3):
                    n = s["n"][b] + 2 * self.g[b]
                    i = self.index(e, a, b, b == a)
                    ok = ok & ((i >= 2) & (i <= n - 4) if b == a else (i >= 3) & (i <= n - 4))
                tl, el = self.visc_low(W, a)
                tau = [torch.where(ok, x, y) for x, y in zip(tau, tl)]
                e = torch.where(ok, e, el)
            F = [F[0]] + [F[1 + c] - tau[c] for c in range(3)] + [F[4] - e]
        return F

    def inner(self, q):
        for a in range(self.dim):
            q = self.cut(q, a, self.g[a], self.s["n"][a])
        return q

    def residual(self, q):
        W = self.prim(q)
        R = [0.0] * (self.dim + 2)
        for a in range(self.dim):
            F = self.flux(W, a)
            met = self.s["dt"] * self.vol / self.s["h"][a]
            for l in range(self.dim + 2):
                f = F[l]
                R[l] = R[l] + met * (self.cut(f, a, 1, self.s["n"][a]) - self.cut(f, a, 0, self.s["n"][a]))
        return torch.stack(R)

    def step(self):
        q, inn = self.q, self.inner
        if self.s["rk"] == 3:
            q1 = q.clone()
            inn(q1).sub_(self.residual(q))
            self.fill(q1)
            q2 = q1.clone()
            inn(q2).copy_(0.75 * inn(q) + 0.25 * inn(q1) - 0.25 * self.residual(q1))
            self.fill(q2)
            inn(q).copy_((2.0 * inn(q2) + inn(q) - 2.0 * self.residual(q2)) / 3.0)
        else:
            acc, src = 0.0, q
            for c1, c2 in ((0.5, 1.0), (0.5, 2.0), (1.0, 2.0)):
                r = self.residual(src)
                src = q.clone()
                inn(src).sub_(c1 * r)
                acc = acc + c2 * r
                self.fill(src)
            inn(q).sub_((acc + self.residual(src)) / 6.0)
        self.fill(q)

    def history(self):
        q = self.q
        r = self.J * q[0]
        v = [q[1 + a] / q[0] for a in range(3)]
        p = (self.s["gamma"] - 1.0) * (self.J * q[4] - 0.5 * r * sum(x * x for x in v))
        d = lambda c, a: ((self.shift(v[c], a, 3) - self.shift(v[c], a, -3)) / 60.0  # noqa: E731
                          - 0.15 * (self.shift(v[c], a, 2) - self.shift(v[c], a, -2))
                          + 0.75 * (self.shift(v[c], a, 1) - self.shift(v[c], a, -1))) / self.s["h"][a]
        om = (d(2, 1) - d(1, 2)) ** 2 + (d(0, 2) - d(2, 0)) ** 2 + (d(1, 0) - d(0, 1)) ** 2
        i = self.inner
        return np.array([float(i(0.5 * r * sum(x * x for x in v)).mean()),
                         float(i(r * torch.log(p * r ** -self.s["gamma"])).mean()), float(i(0.5 * r * om).mean())])


def exact(case, seed):
    solves = _solves(case)
    if sum(float(np.prod(s["n"])) for s in solves) > EXACT_CELLS:
        return None
    out = []
    for i, s in enumerate(solves):
        x = _Exact(s, _field(s, seed + 1000 * i, _device()))
        x.fill(x.q)
        for _ in range(case["steps"]):
            x.step()
        out.append(x)
    if case["family"] in ("ensemble", "les_batch"):
        return _outputs(case, [x.q for x in out])
    d = _parts(out[0].q)
    if case.get("history"):
        d["history"] = out[0].history()
    return d
