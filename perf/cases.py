"""The solves that programs of this framework run, as measurable cases.

Each case builds its mesh, controls and seeded start once (``prepare``) and
then runs one pass of a program through the public entry points (``run``): a
restart state goes to the device, a stretch of the solve runs, and the state,
the history or the sensitivities come back.  Kinds:

* ``steady``    -- run_steady from a restart state: cycles with the residuals
  and forces read after each, as every steady run does;
* ``unsteady``  -- run_unsteady (dual time stepping) with a fixed number of
  cycles per physical step;
* ``batch``     -- many flow conditions on one mesh through Batch.run;
* ``smoother``  -- relaxation steps of the finest level alone
  (do_time_iterations, the call the reference's driver makes);
* ``residual``  -- residual_fwd and residual_vjp, the forward and backward
  product of the central residual on host arrays;
* ``adjoint``   -- adjoint_solve: GMRES steps and the geometry sweep.

The meshes are the repository's generators' at sizes of its tests, benchmark
and profiles, and odd ones between.  Meshes depend on the sizes alone and are
built once per process; everything else is made anew by ``prepare``.
"""
import functools
import math

import numpy as np
import torch

import flite3d_b200 as F
from flite3d_b200.solver import Batch, run_steady, run_unsteady

BUMP_HEIGHT = 0.05

# the flow models, by the controls that a deck sets
MODELS = {
    # Euler, central flux with JST dissipation (the reference's default)
    "euler": dict(ReynoldsNumber=0.0, MachNumber=0.5, alpha=0.0, CFLNumber=2.0, fluxType=1),
    # laminar Navier-Stokes with adiabatic walls, the benchmark's workload
    "laminar": dict(ReynoldsNumber=5000.0, MachNumber=0.5, alpha=0.0, CFLNumber=2.0, fluxType=1,
                    wallsAreIsentropic=1, viscosityScheme=1),
    # the same with the compact viscous stencil
    "laminar2": dict(ReynoldsNumber=5000.0, MachNumber=0.5, alpha=0.0, CFLNumber=1.0, fluxType=1,
                     wallsAreIsentropic=1, viscosityScheme=2),
    # the same with FP32 flux increments over an FP64 anchor
    "mixed": dict(ReynoldsNumber=5000.0, MachNumber=0.5, alpha=0.0, CFLNumber=2.0, fluxType=1,
                  wallsAreIsentropic=1, viscosityScheme=1, precision=1),
    # Euler with the reconstructed HLLC flux of the example deck
    "hllc": dict(ReynoldsNumber=0.0, MachNumber=0.5, alpha=0.0, CFLNumber=1.0, fluxType=4, HLLCFluxOrder=2,
                 Automaticlipping=1, GradientMethod=1),
    # Euler with the Roe flux, Van Albada reconstruction and five stages
    "upwind": dict(ReynoldsNumber=0.0, MachNumber=0.5, alpha=0.0, CFLNumber=2.0, fluxType=3, reconstruction=1,
                   rungeKuttaStages=5, secondOrderDissipationFactor=0.0, fourthOrderDissipationFactor=0.0),
    # Spalart-Allmaras RANS with the reconstructed HLLC flux
    "rans": dict(ReynoldsNumber=6.0e6, MachNumber=0.8, alpha=1.25, CFLNumber=1.0, fluxType=4, HLLCFluxOrder=2,
                 Automaticlipping=1, GradientMethod=1, turbulenceModel=1, wallsAreIsentropic=1),
}


def listed():
    return [
        # the reference-sized Euler case that a user starts with: 14 thousand
        # nodes, where launches and the host's reads after each cycle count
        dict(name="euler_small", kind="steady", model="euler", mesh="bump", nx=48, ny=16, nz=16, levels=3, scheme=3,
             cycles=25),
        # a ragged mid-sized Euler mesh with the example deck's HLLC flux, V-cycle
        dict(name="hllc_ragged", kind="steady", model="hllc", mesh="bump", nx=83, ny=29, nz=31, levels=3, scheme=1,
             cycles=10),
        # laminar flow at the batch's smallest mesh, the everyday size
        dict(name="laminar_mid", kind="steady", model="laminar", mesh="bump", nx=120, ny=40, nz=40, levels=4,
             scheme=3, cycles=20),
        # the benchmark's workload: 2.1 million nodes
        dict(name="laminar_large", kind="steady", model="laminar", mesh="bump", nx=264, ny=88, nz=88, levels=4,
             scheme=3, cycles=8),
        # the mixed-precision option on the second benchmark mesh
        dict(name="mixed_large", kind="steady", model="mixed", mesh="bump", nx=192, ny=64, nz=64, levels=4, scheme=3,
             cycles=8),
        # turbulent flow over a wing section: O-grid with thin wall layers
        dict(name="rans_wing", kind="steady", model="rans", mesh="naca", nx=100, ny=60, nz=120, levels=5, scheme=3,
             cycles=4),
        # the upwind extension, W-cycle
        dict(name="upwind_mid", kind="steady", model="upwind", mesh="bump", nx=120, ny=40, nz=40, levels=3, scheme=2,
             cycles=5),
        # time-accurate laminar flow, two physical steps
        dict(name="unsteady_ragged", kind="unsteady", model="laminar", mesh="bump", nx=97, ny=33, nz=31, levels=4,
             scheme=3, cycles=6, steps=2),
        # a polar of sixteen conditions on one small mesh
        dict(name="polar_small", kind="batch", model="euler", mesh="bump", nx=48, ny=16, nz=16, levels=3, scheme=3,
             cycles=12, conditions=16),
        # relaxation of the fine level alone
        dict(name="smoother_large", kind="smoother", model="laminar", mesh="bump", nx=192, ny=64, nz=64, levels=1,
             scheme=3, cycles=6),
        # forward and backward product of the residual on host arrays
        dict(name="residual_mid", kind="residual", model="euler", mesh="bump", nx=121, ny=39, nz=41, levels=1,
             scheme=3, cycles=1),
        # lift sensitivities: GMRES on the transposed smoother
        dict(name="adjoint_small", kind="adjoint", model="laminar", mesh="bump", nx=48, ny=16, nz=16, levels=3,
             scheme=3, cycles=120),
    ]


# per kind: the models it is run with, the largest mesh (nodes) and cycles
_RANGES = {
    "steady": (("euler", "laminar", "laminar2", "mixed", "hllc", "upwind", "rans"), 1.0e6, (4, 24)),
    "unsteady": (("euler", "laminar"), 4.0e5, (3, 8)),
    "batch": (("euler", "mixed"), 4.0e4, (6, 16)),
    "smoother": (("euler", "laminar"), 1.0e6, (2, 8)),
    "residual": (("euler",), 4.0e5, (1, 1)),
    "adjoint": (("euler", "laminar"), 4.0e4, (60, 140)),
}


def draw(rng):
    kind = rng.choice(["steady"] * 4 + ["unsteady", "batch", "smoother", "residual", "adjoint"])
    models, most, (c0, c1) = _RANGES[kind]
    model = rng.choice(models)
    n = math.exp(rng.uniform(math.log(8.0e3), math.log(most)))
    m = max(8, round((n / 3.0) ** (1.0 / 3.0)))
    levels = 1 if kind in ("smoother", "residual") else rng.choice([3, 4])
    c = dict(kind=kind, model=model, levels=levels, scheme=rng.choice([1, 3, 3, 2]), cycles=rng.randint(c0, c1))
    if model == "rans":
        c.update(mesh="naca", nx=2 * max(12, round(0.45 * m * rng.uniform(0.9, 1.2))), ny=max(45, m),
                 nz=max(6, round(1.2 * m * rng.uniform(0.8, 1.1))), scheme=3)
        c["cycles"] = min(c["cycles"], 6)
    else:
        c.update(mesh="bump", nx=max(16, round(3 * m * rng.uniform(0.85, 1.15))), ny=max(8, m + rng.randint(-3, 3)),
                 nz=max(8, m + rng.randint(-3, 3)))
    if n > 2.0e5:
        c["cycles"] = max(2, min(c["cycles"], 8))
    if kind == "unsteady":
        c["steps"] = rng.choice([1, 2, 3])
    if kind == "batch":
        c["conditions"] = rng.choice([4, 7, 16, 20])
    return c


# ---- meshes, controls and starts ------------------------------------------

@functools.lru_cache(maxsize=None)
def _mesh(kind, nx, ny, nz, levels):
    if kind == "naca":
        return F.Mesh.naca0012(nx, ny, nz, first_cell=1.0e-5, growth=1.15, nlayer=40, farfield=20.0, span=1.0,
                               nlevels=levels)
    return F.Mesh.bump_channel(nx, ny, nz, BUMP_HEIGHT, levels)


@functools.lru_cache(maxsize=None)
def _jittered(nx, ny, nz, levels):
    """The bump channel with moved interior nodes (no two edges tie in the
    dissipation's switches, whose derivative the adjoint takes)."""
    base = _mesh("bump", nx, ny, nz, levels)
    x = base.array(1, "coords")
    jit = np.random.default_rng(11).uniform(-1, 1, x.shape) * 0.15 / nz
    jit[:, :base.level(1).n_bnodes] = 0.0
    return base.with_level1_geometry(*base.geometry(x + jit))


def _case_mesh(case):
    if case["kind"] == "adjoint":
        return _jittered(case["nx"], case["ny"], case["nz"], case["levels"])
    return _mesh(case["mesh"], case["nx"], case["ny"], case["nz"], case["levels"])


def _controls(case, **more):
    ctl = dict(MODELS[case["model"]], multigridScheme=case["scheme"], numberOfGridsToUse=case["levels"])
    if case["kind"] == "unsteady":
        ctl.update(flowType=1, physicalTimeStep=0.1)
    return F.default_controls(**{**ctl, **more})


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    v = t.numpy()
    v[...] = a
    return t, v


def prepare(case, seed):
    mesh = _case_mesh(case)
    kind = case["kind"]
    st = dict(case=case, mesh=mesh)
    if kind == "batch":
        rng = np.random.default_rng(seed)
        cond = [(-4.0 + 12.0 * a, 0.3 + 0.5 * b) for a, b in rng.random((case["conditions"], 2))]
        cases = [(_controls(case, alpha=a, MachNumber=m), mesh) for a, m in cond]
        st["batch"] = Batch(cases)
        st["u0"], st["out"], st["keep"] = [], [], []
        for c, m in cases:
            for where in ("u0", "out"):
                t, v = _pinned(F.initial_state(c, m))
                st["keep"].append(t)
                st[where].append(v)
        return st
    c = _controls(case)
    s = F.Solver(c, mesh)
    u0 = F.initial_state(c, mesh, perturb_seed=seed, amplitude=0.01)
    if kind in ("smoother", "residual"):
        # a developed field: every component varies from node to node
        r = np.random.default_rng(seed).uniform(-1.0, 1.0, (4, u0.shape[1]))
        u0[1] *= 1.0 + 0.03 * r[0]
        u0[2] += 0.02 * r[1]
        u0[3] += 0.015 * r[2]
        u0[4] *= 1.0 + 0.01 * r[3]
    st.update(solver=s, controls=c)
    st["keep"], st["u0"] = _pinned(u0)
    st["keep_out"], st["out"] = _pinned(np.zeros_like(u0))
    if kind == "residual":
        st["rbar"] = np.random.default_rng(seed + 1).standard_normal(u0.shape)
    if kind == "adjoint":
        # the flow that is differentiated: a stretch of its solve
        s.set_state(st["u0"])
        s.start()
        for it in range(1, 301):
            s.cycle(it)
    return st


def run(st):
    case = st["case"]
    kind, n = case["kind"], case["cycles"]
    if kind == "batch":
        b = st["batch"]
        for s, u in zip(b.cases, st["u0"]):
            s.set_state(u)
            s.start()
        cyc, red = b.run(orders=50.0, max_cycles=n)
        return dict(cycles=cyc, reduction=red, state=[s.get_state(out=o) for s, o in zip(b.cases, st["out"])])
    s = st["solver"]
    if kind == "residual":
        return dict(residual=s.residual_fwd(st["u0"]), product=s.residual_vjp(st["u0"], st["rbar"]))
    if kind == "adjoint":
        r = s.adjoint_solve("CL", tol=1e-12, max_iter=n)
        return dict(J=r["J"], side=r["side_w_bar"], boundary=r["bnd_w_bar"], volume=r["volume_bar"])
    s.set_state(st["u0"])
    s.start()
    if kind == "smoother":
        s.do_time_iterations(1, nsteps=n)
        return dict(state=s.get_state(out=st["out"]))
    if kind == "unsteady":
        hist = run_unsteady(s, case["steps"], n)
    else:
        hist = run_steady(s, orders=50.0, max_cycles=n)
    return dict(history=np.array([h[1] for h in hist]), state=s.get_state(out=st["out"]))


# ---- the work of one pass -------------------------------------------------

def _sweeps(case):
    """Per level (finest first): the edge sweeps of the flux (RK stages and
    restriction steps) and of the dissipation, time step and viscous terms
    in one pass, from the cycle's relaxations and transfers."""
    g, scheme = case["levels"], case["scheme"]
    relax, restrict, prolong = [0] * g, [0] * g, [0] * g

    def down(top):
        for j in range(top, g):
            relax[j - 1] += 1
            restrict[j - 1] += 1
        relax[g - 1] += 1

    def up(to, smooth):
        for j in range(g, to, -1):
            prolong[j - 2] += 1
            if smooth:
                relax[j - 2] += 1

    if g == 1 or case["kind"] == "smoother":
        relax[0] += 1
    elif scheme == 1:
        down(1)
        up(1, True)
    elif scheme == 2:
        nsw, top = (1 if g <= 2 else 2 * g - 4), 1
        for i in range(1, nsw + 1):
            down(top)
            top = (g - 1 if g > 2 else g) if top == 1 else (top - 1 if i <= nsw // 2 else top + 1)
            up(top, True)
        up(1, True)
    else:
        top = 1
        for _ in range(g - 1):
            down(top)
            top = g - 1 if top == 1 else top - 1
            up(top, False)
    return relax, restrict, prolong


def work(case):
    nodes = (case["nx"] + (0 if case["mesh"] == "naca" else 1)) * (case["ny"] + 1) * (case["nz"] + 1)
    edges = 7 * nodes
    if case["kind"] == "residual":
        # both products read the state, the coefficients and the other input once
        return dict(bytes=2 * (40 + 40) * nodes + 2 * 32 * edges, flops=2 * 90 * edges)
    model = case["model"]
    stages = 5 if model == "upwind" else 3
    flux = {"hllc": 400, "rans": 400, "upwind": 250}.get(model, 70)     # operations of one edge flux
    viscous = model in ("laminar", "laminar2", "mixed", "rans")
    nvar = 6 if model == "rans" else 5
    repeats = case["cycles"] * case.get("steps", 1) * case.get("conditions", 1)
    if case["kind"] == "adjoint":
        # a product reverses one smoother iteration: its sweeps once more, and
        # the Krylov vectors (50 at most, half of them on average) twice
        sweep = 32 * edges + 2 * 8 * 6 * nodes
        return dict(bytes=repeats * (7 * sweep + 2 * 25 * 48 * nodes), flops=repeats * (500 * edges + 600 * nodes))
    relax, restrict, prolong = _sweeps(case)
    b = f = 0.0
    for lv in range(case["levels"]):
        n, e = nodes / 8.8 ** lv, edges / 7.5 ** lv
        extra = 1 + (2 if viscous else 0) + (0 if model in ("hllc", "upwind", "rans") else 1)
        # flux sweep: coefficients and indices; state, previous state, dissipation, dt and V in, state out
        fb, ff = 32 * e + 8 * (4 * nvar + 2) * n, flux * e
        # time step, dissipation and viscous sweeps: coefficients, two node fields in, one out
        db, df = extra * (32 * e + 3 * 8 * nvar * n), extra * 40 * e
        nflux = stages * relax[lv] + restrict[lv] + (restrict[lv - 1] if lv else 0)
        ndiss = relax[lv] + restrict[lv] + (restrict[lv - 1] if lv else 0)
        b += nflux * fb + ndiss * db + (restrict[lv] + prolong[lv]) * 8 * 2 * nvar * n
        f += nflux * ff + ndiss * df
    return dict(bytes=repeats * b, flops=repeats * f)


# ---- plain 64-bit values --------------------------------------------------
# The single-level terms of the scheme in torch, written from the scheme's
# definition: edges scatter to their two nodes.  Whole multigrid runs and
# sensitivities have no short independent form; they are held to the bound of
# their type.

class _Level:
    def __init__(self, mesh):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda name: torch.from_numpy(np.ascontiguousarray(mesh.array(1, name))).to(dev)
        idx, bidx = t("side_idx").long() - 1, t("bnd_idx").long()
        self.i1, self.i2, self.w = idx[0], idx[1], t("side_w")
        self.b1, self.b2, self.bind, self.bw = bidx[0] - 1, bidx[1] - 1, bidx[2], t("bnd_w")
        self.V = t("volume")
        self.n = self.V.shape[0]
        ones = torch.ones_like(self.w[0])
        self.conn = self.scatter(ones, ones)
        a = self.bscatter(-self.bw, -self.bw)
        nrm = a.square().sum(0).sqrt()
        self.normal = torch.where(nrm > 1e-10, a / nrm.clamp_min(1e-300), torch.zeros_like(a))
        self.cls = torch.zeros(self.n, dtype=torch.long, device=dev)
        reg, ind = mesh.array(1, "node_reg"), mesh.array(1, "node_ind")
        for k in range(1, 10):
            lo, hi = int(reg[2 * (k - 1)]), int(reg[2 * k - 1])
            if hi >= lo:
                self.cls[torch.from_numpy(ind[lo - 1:hi].astype(np.int64) - 1).to(dev)] = k

    def _add(self, i, a, j, b):
        out = torch.zeros(a.shape[:-1] + (self.n,), dtype=torch.float64, device=a.device)
        return out.index_add(-1, i, a).index_add(-1, j, b)

    def scatter(self, a, b):
        return self._add(self.i1, a, self.i2, b)

    def bscatter(self, a, b):
        return self._add(self.b1, a, self.b2, b)


def _pressure(c, u):
    return ((c.gamma - 1.0) * (u[4] - 0.5 * u[1:4].square().sum(0) / u[0])).clamp_min(0.1)


def _physical(u, p, n):
    """The flux of a state through unit normals n."""
    v = u[1:4] / u[0]
    vn = (v * n).sum(0)
    return torch.cat([(u[0] * vn)[None], p * n + u[1:4] * vn, ((u[4] + p) * vn)[None]])


def _farfield(c, u, p, n, inf):
    """Roe flux between a state and the freestream."""
    g1 = c.gamma - 1.0
    ro, vo, eo, po = inf[0], torch.tensor(inf[1:4], dtype=torch.float64, device=u.device)[:, None], inf[4], inf[5]
    v, hl = u[1:4] / u[0], (u[4] + p) / u[0]
    er, hr, un = eo * ro, eo + po / ro, (vo * n).sum(0)
    fr = torch.cat([(ro * un)[None], po * n + ro * vo * un, ((er + po) * un)[None]])
    di = (ro / u[0]).sqrt()
    vi, hi = (di * vo + v) / (di + 1.0), (di * hr + hl) / (di + 1.0)
    q = 0.5 * vi.square().sum(0)
    c2 = (g1 * (hi - q)).clamp_min(1e-5)
    ci, ucp = c2.sqrt(), (vi * n).sum(0)
    du = torch.cat([(ro - u[0])[None], ro * vo - u[1:4], (er - u[4])[None]])
    l1, l2, l3 = (ucp + ci).abs(), (ucp - ci).abs(), ucp.abs()
    s1, s2 = 0.5 * (l1 + l2), 0.5 * (l1 - l2)
    a1 = g1 * (q * du[0] - (vi * du[1:4]).sum(0) + du[4])
    a2 = -ucp * du[0] + (du[1:4] * n).sum(0)
    k1, k2 = (s1 - l3) * a1 / c2 + s2 * a2 / ci, s2 * a1 / ci + (s1 - l3) * a2
    d = torch.cat([(l3 * du[0] + k1)[None], l3 * du[1:4] + k1 * vi + k2 * n, (l3 * du[4] + k1 * hi + k2 * ucp)[None]])
    return 0.5 * (fr + _physical(u, p, n)) - 0.5 * d


def _residual(c, g, u):
    p = _pressure(c, u)
    v, h = u[1:4] / u[0], u[4] + p

    def one(i):
        un = (g.w * v[:, i]).sum(0)
        return torch.cat([(u[0, i] * un)[None], u[1:4, i] * un + p[i] * g.w, (h[i] * un)[None]])

    f = one(g.i1) + one(g.i2)
    r = g.scatter(f, -f)
    area = g.bw.square().sum(0).sqrt()
    n = g.bw / area
    f1, f2 = (_physical(u[:, b], p[b], n) for b in (g.b1, g.b2))
    for k in (3, 4):
        at = g.bind == k
        if bool(at.any()):
            inf = [float(x) for x in c.inflowField[6 * (k - 3):6 * (k - 3) + 6]]
            f1, f2 = (torch.where(at, _farfield(c, u[:, b], p[b], n, inf), f) for b, f in ((g.b1, f1), (g.b2, f2)))
    return r + g.bscatter(area * (3.0 * f1 + f2), area * (f1 + 3.0 * f2))


def _time_step(c, g, u, p, mu):
    def speeds(w, i):
        return (w * u[1:4, i]).sum(0).abs() / u[0, i] + ((c.gamma * p[i] / u[0, i]).clamp_min(0.001)
                                                        * w.square().sum(0)).sqrt()

    a = g.scatter(speeds(g.w, g.i1), speeds(g.w, g.i2))
    s1, s2 = speeds(g.bw, g.b1), speeds(g.bw, g.b2)
    a = a + g.bscatter(2.0 * s1 + s2, s1 + 2.0 * s2)
    h = torch.zeros_like(a)
    if c.ReynoldsNumber > 0:
        k = 2.0 * mu.clamp_min(1.0 / c.ReynoldsNumber) / u[0]
        al, bl = g.w.square().sum(0), g.bw.square().sum(0)
        h = g.scatter(k[g.i2] * al, k[g.i1] * al)
        d1, d2 = k[g.b1] * bl, k[g.b2] * bl
        h = h + g.bscatter(2.0 * d1 + d2, d1 + 2.0 * d2)
    return 0.5 / (a / g.V + h / g.V.square())


def _jst(c, g, u, p, dt):
    q = torch.cat([u[:4], (u[4] + p)[None]])
    d = q[:, g.i1] - q[:, g.i2]
    lap = g.scatter(-d, d) / g.conn
    dp, sp = p[g.i1] - p[g.i2], p[g.i1] + p[g.i2]
    sensor = 12.0 * (g.scatter(-dp, dp) / g.scatter(sp, sp)).abs()
    k = g.V / dt
    d0 = torch.minimum(k[g.i1], k[g.i2]) / (g.conn[g.i1] + g.conn[g.i2])
    e2 = d0 * c.secondOrderDissipationFactor * torch.maximum(sensor[g.i1], sensor[g.i2])
    e4 = (d0 * c.fourthOrderDissipationFactor - e2).clamp_min(0.0)
    t = -(lap[:, g.i1] - lap[:, g.i2]) * e4 + (u[:, g.i1] - u[:, g.i2]) * e2
    return g.scatter(t, -t)


def _viscous(c, g, u, p):
    """The viscous term as it is added to the dissipation, and the viscosity."""
    ratio = c.gamma / (c.gamma - 1.0)
    T = ratio * p / u[0]
    q = torch.cat([u[1:4] / u[0], T[None]])
    s, sb = q[:, g.i1] + q[:, g.i2], q[:, g.b1] + q[:, g.b2]
    grad = torch.stack([g.scatter(s * g.w[a], -s * g.w[a]) + g.bscatter((2.0 * q[:, g.b1] + sb) * g.bw[a],
                                                                      (2.0 * q[:, g.b2] + sb) * g.bw[a])
                        for a in range(3)]) / g.V                 # [direction][component]
    tc, tin = (c.gamma - 1.0) * c.MachNumber ** 2, c.inflowTemperature
    T = T.clamp_min(0.001)
    mu = (tc * T) ** 1.5 * (tin + 198.6) / (tc * tin * T + 198.6) / c.ReynoldsNumber
    vel = grad[:, :3]
    div = vel[0, 0] + vel[1, 1] + vel[2, 2]
    eye = torch.eye(3, dtype=torch.float64, device=u.device)[:, :, None]
    tau = mu * (vel + vel.transpose(0, 1) - (2.0 / 3.0) * div * eye)
    heat = mu / c.PrandtlNumber * grad[:, 3]
    heat = torch.where(g.cls == 1, heat - (heat * g.normal).sum(0) * g.normal, heat)
    row = torch.cat([tau, ((tau * q[:3]).sum(1) + heat)[:, None]], 1)  # [direction][4]

    def through(w, i):
        return (w[:, None] * row[:, :, i]).sum(0)

    f = through(g.w, g.i1) + through(g.w, g.i2)
    acc = g.scatter(f, -f)
    on = ((g.bind != 2) & (g.bind != 9)).to(torch.float64)
    f1, f2 = through(g.bw, g.b1) * on, through(g.bw, g.b2) * on
    acc = acc + g.bscatter(3.0 * f1 + f2, f1 + 3.0 * f2)
    return torch.cat([torch.zeros_like(acc[:1]), -acc]), mu


def _slip(x, n, at):
    m = x[1:4] - (x[1:4] * n).sum(0) * n
    return torch.cat([x[:1], torch.where(at, m, x[1:4]), x[4:]])


def _outer(c, g, u, p):
    for k in (3, 4):
        inf = [float(x) for x in c.inflowField[6 * (k - 3):6 * (k - 3) + 6]]
        v = torch.tensor(inf[1:4], dtype=torch.float64, device=u.device)[:, None]
        into = (v * g.normal).sum(0) > 0.0
        e_in = p / (c.gamma - 1.0) + 0.5 * float(v.square().sum()) * inf[0]
        if c.MachNumber > 1.0:
            e_in = torch.full_like(p, inf[4] * inf[0])
        inflow = torch.cat([torch.full_like(u[:1], inf[0]), (v * inf[0]).expand(3, g.n), e_in[None]])
        e_out = inf[5] / (c.gamma - 1.0) + 0.5 * u[1:4].square().sum(0) / u[0]
        out = torch.cat([u[:4], (e_out if c.MachNumber < 1.0 else u[4])[None]])
        u = torch.where(g.cls == k, torch.where(into, inflow, out), u)
    return u


def _conditions(c, g, u):
    """The solution conditions of static walls and symmetry planes."""
    wall = g.cls == 1
    if c.ReynoldsNumber > 0:
        u = torch.cat([u[:1], torch.where(wall, torch.zeros_like(u[1:4]), u[1:4]), u[4:]])
        if not c.wallsAreIsentropic:
            u = torch.cat([u[:4], torch.where(wall, u[0] * c.inflowTemperature / c.gamma, u[4])[None]])
        return _slip(u, g.normal, g.cls == 2)
    return _slip(u, g.normal, wall | (g.cls == 2))


def _relax(c, g, u, mu):
    """One relaxation step of the finest level: (state, viscosity)."""
    u0, p = u, _pressure(c, u)
    dt = _time_step(c, g, u, p, mu)
    diss = _jst(c, g, u, p, dt)
    if c.ReynoldsNumber > 0:
        term, mu = _viscous(c, g, u, p)
        diss = diss + term
    wall = g.cls == 1
    for rk in (0.6, 0.6, 1.0):
        p = _pressure(c, u)
        r = dt * (_residual(c, g, u) + diss) / g.V
        if c.ReynoldsNumber > 0:
            r = torch.cat([r[:1], torch.where(wall, torch.zeros_like(r[1:4]), r[1:4]), r[4:]])
            if not c.wallsAreIsentropic:
                r = torch.cat([r[:4], torch.where(wall, torch.zeros_like(r[4]), r[4])[None]])
            r = _slip(r, g.normal, g.cls == 2)
        else:
            r = _slip(r, g.normal, wall | (g.cls == 2))
        d = c.CFLNumber * rk * r
        most = c.maxIncrementFactor
        rho = torch.where((d[0] / u0[0]).abs() < most, u0[0] - d[0], u0[0] - torch.sign(d[0]) * most * u0[0])
        u = torch.cat([rho.clamp_min(c.minimumDensity)[None], u0[1:] - d[1:]])
        u = _conditions(c, g, u)
        u = _outer(c, g, torch.cat([u[:1].clamp_min(c.minimumDensity), u[1:]]), p)
    return u, mu


def exact(case, seed):
    if case["kind"] not in ("smoother", "residual"):
        return None
    st = prepare(case, seed)
    c, g = st["controls"], _Level(_case_mesh(case))
    u = torch.from_numpy(np.array(st["u0"])).to(g.V.device)
    if case["kind"] == "residual":
        u.requires_grad_(True)
        r = _residual(c, g, u)
        (product,) = torch.autograd.grad(r, u, torch.from_numpy(st["rbar"]).to(r.device))
        return dict(residual=r.detach(), product=product)
    mu = torch.full_like(g.V, 1.0 / c.ReynoldsNumber if c.ReynoldsNumber > 0 else 0.0)
    u = _conditions(c, g, u)
    for _ in range(case["cycles"]):
        u, mu = _relax(c, g, u, mu)
    return dict(state=u)
