"""Performance cases: the work that programs give this framework, and what it should answer.

A pass of an "advance" case is what a solver run does between two outputs: upload the state, take a
number of explicitLoop steps, read the state back (the asynchronous transfers, pinned buffers).
A pass of the "train" case is one epoch of the learned equilibrium surrogate's training.

`exact` restates the solver in plain torch, 64 bits, on the mesh arrays that `prepare` has too.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from fooskagpu_b200 import cases as physics
from fooskagpu_b200 import meshgen
from fooskagpu_b200.api import Mesh, Solver, Surrogate

DEVICE = "cuda:0"


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the periodic Taylor-Green vortex (WALE LES, heat conduction) of the benchmark: a mesh of the
        # size the tests use (launches and latency count), a development size, the benchmark's own
        dict(name="tgv_tiny", kind="advance", problem="tgv", nx=8, ny=8, nz=8, precision="mixed", steps=4, dt_every=2,
             surrogate=False, monitor=False, stages=False),
        dict(name="tgv_small", kind="advance", problem="tgv", nx=40, ny=40, nz=40, precision="mixed", steps=10,
             dt_every=10, surrogate=False, monitor=False, stages=False),
        dict(name="tgv_large", kind="advance", problem="tgv", nx=128, ny=128, nz=128, precision="mixed", steps=10,
             dt_every=10, surrogate=False, monitor=False, stages=False),
        # the same vortex in full FP64, the path that results are checked against
        dict(name="tgv_fp64", kind="advance", problem="tgv", nx=96, ny=96, nz=96, precision="fp64", steps=5,
             dt_every=5, surrogate=False, monitor=False, stages=False),
        # Sod tube on 480,000 jittered tets: inviscid, FP64, slip walls
        dict(name="sod_fp64", kind="advance", problem="sod", nx=200, ny=20, nz=20, precision="fp64", steps=10,
             dt_every=1, surrogate=False, monitor=False, stages=False),
        # bubble collapse on a coarse graded ball, watched step by step (probe), as a parameter study does
        dict(name="bubble_watched", kind="advance", problem="bubble", nx=24, ny=24, nz=24, precision="mixed", steps=5,
             dt_every=1, surrogate=False, monitor=True, stages=False),
        # bubble collapse at production size: stiff water, about nine thermal Newton iterations per cell
        dict(name="bubble_large", kind="advance", problem="bubble", nx=57, ny=57, nz=57, precision="mixed", steps=5,
             dt_every=1, surrogate=False, monitor=False, stages=False),
        # liquid jet into pressurised gas on prisms and tets: walls, inlet, outlet, dt every step
        dict(name="jet", kind="advance", problem="jet", nx=72, ny=72, nz=100, precision="mixed", steps=4, dt_every=1,
             surrogate=False, monitor=False, stages=False),
        # tets, pyramids, prisms and hexes in one mesh, driven by the stage functions one by one as the
        # reference's explicitLoop drives its own
        dict(name="stage_calls", kind="advance", problem="elements", nx=23, ny=19, nz=17, precision="mixed", steps=3,
             dt_every=3, surrogate=False, monitor=False, stages=True),
        # evaporating liquid / vapour mixture, a third of the cells in the Gibbs Newton, FP64
        dict(name="mixture_fp64", kind="advance", problem="mixture", nx=61, ny=67, nz=59, precision="fp64", steps=3,
             dt_every=1, surrogate=False, monitor=False, stages=False),
        # the same mixture in mixed precision with the learned surrogate in front of the Newton
        dict(name="mixture_surrogate", kind="advance", problem="mixture", nx=64, ny=64, nz=64, precision="mixed",
             steps=3, dt_every=1, surrogate=True, monitor=False, stages=False),
        # training the surrogate: loss and gradient of one batch, then an epoch of Adam steps
        dict(name="train", kind="train", samples=65536, batch=4096),
    ]


def draw(rng):
    kind = rng.choice(["tgv", "tgv", "sod", "bubble", "jet", "elements", "mixture", "mixture", "train"])
    if kind == "train":
        batch = int(round(2 ** rng.uniform(9, 14)))
        return dict(kind="train", samples=batch * rng.randint(4, 12) + rng.randint(0, 31), batch=batch)
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))   # noqa: E731
    section = rng.randint(5, 20)
    nx, ny, nz = {
        "tgv": lambda: (log(7, 110), log(7, 110), log(7, 110)),
        "sod": lambda: (10 * section, section, section),
        "bubble": lambda: (log(12, 56),) * 3,
        "jet": lambda: (log(24, 72),) * 2 + (2 * log(5, 50),),
        "elements": lambda: (rng.randint(6, 24), rng.randint(6, 20), rng.randint(6, 20)),
        "mixture": lambda: (log(9, 70), log(9, 70), log(9, 70)),
    }[kind]()
    precision = rng.choice(["mixed", "mixed", "fp64"])
    steps = rng.randint(2, 4)
    return dict(kind="advance", problem=kind, nx=nx, ny=ny, nz=nz, precision=precision, steps=steps,
                dt_every=1 if kind in ("sod", "bubble", "jet") else rng.choice([1, steps]),
                surrogate=kind == "mixture" and rng.random() < 0.5, monitor=rng.random() < 0.25,
                stages=rng.random() < 0.2)


# ---------------------------------------------------------------- meshes, parameters, initial states
_meshes: dict = {}


def _mesh(case):
    """The case's mesh (handle, .neu-order arrays): read once by a program and kept."""
    key = (case["problem"], case["nx"], case["ny"], case["nz"])
    if key not in _meshes:
        kind, nx, ny, nz = key
        periodic = (0.0, 0.0, 0.0)
        if kind == "tgv":
            L = 2 * math.pi
            nm, periodic = meshgen.box_hexes(nx, ny, nz, L=(L, L, L), side_bc={}, shuffle=True), (L, L, L)
        elif kind == "sod":
            nm = meshgen.box_tets(nx, ny, nz, L=(1.0, 0.1, 0.1), jitter=0.1,
                                  side_bc={s: "slip" for s in ("x0", "x1", "y0", "y1", "z0", "z1")})
        elif kind == "bubble":
            nm = meshgen.ball_tets(nx)
        elif kind == "jet":
            nm = meshgen.jet_cylinder(n=nx, nz_prism=nz // 2, nz_tet=nz // 2)
        elif kind == "elements":
            nm = meshgen.box_mixed(nx, ny, nz, L=(nx * 1e-3, ny * 1e-3, nz * 1e-3),
                                   side_bc={"x0": "inlet", "x1": "outlet", "y0": "wall", "y1": "slip",
                                            "z0": "symmetry", "z1": "slip"})
        else:
            nm = meshgen.box_hexes(nx, ny, nz, L=(nx * 1e-3, ny * 1e-3, nz * 1e-3), shuffle=True)
        m = Mesh.build(nm.nodes, nm.elems, nm.bcs, periodic=periodic, gpu=True)
        _meshes[key] = (m, m.arrays())
    return _meshes[key]


def _parameters(case):
    kind = case["problem"]
    c = {"tgv": physics.tgv_case, "sod": physics.sod_case, "jet": physics.jet_case,
         "bubble": lambda: physics.water_vapour_case(limiter=0)}.get(kind, physics.reference_case)()
    c.rkSteps = 3
    c.adaptDtItr = case["dt_every"]
    if kind == "sod":
        c.hllcEnergyFix = 1      # the full tube runs to its end only with it
        c.relaxFlag = 1          # one gas: no phase change
    # walls hold S* = 0 exactly, where round-off would pick the branch of a discontinuous flux
    c.hllcTieTol = 1e-4 if case["precision"] == "mixed" else 1e-9
    return c


def _initial(case, c, x, seed):
    rng = np.random.default_rng(seed)
    kind = case["problem"]
    if kind == "tgv":
        return physics.tgv_ic(c, x + rng.uniform(0, 2 * math.pi, 3))
    if kind == "sod":
        # the diaphragm on one of the mesh's planes
        U = physics.sod_ic(c, x, x0=rng.integers(round(0.4 * case["nx"]), round(0.6 * case["nx"])) / case["nx"])
        return U * (1.0 + 0.01 * np.sin(20 * x[:, :1] + rng.uniform(0, 6)) * (np.arange(10) > 0))
    if kind == "bubble":
        spacing = meshgen.ball_spacing(case["nx"], 1e-3)
        return physics.bubble_ic(c, x - rng.uniform(-2e-5, 2e-5, 3), R0=rng.uniform(0.95e-3, 1.1e-3),
                                 width=1.5 * spacing, u_wall=rng.uniform(-10, -5))
    if kind == "jet":
        # the jet has entered: a liquid column with a soft surface, the gas around it at rest
        D, length = 0.2e-3, rng.uniform(2e-3, 6e-3)
        r = np.hypot(x[:, 0], x[:, 1])
        inside = 0.25 * (1 - np.tanh((r - 0.5 * D) / (0.4 * D))) * (1 - np.tanh((x[:, 2] - length) / (2 * D)))
        alpha = c.avfMin + (1 - 2 * c.avfMin) * inside
        p, T = np.full(len(x), c.inletP) * rng.uniform(0.99, 1.01), c.inletT
        rl, rg = physics.rho_of_pT(c, 0, p, T), physics.rho_of_pT(c, 1, p, T)
        z = np.zeros(len(x))
        w = rng.uniform(150, 200) * inside
        return physics.prim_to_cons(c, alpha, rl, rg, z, z, w, p, p, (1 - alpha) * rg)
    return physics.perturbed_two_phase_ic(c, x, seed=seed, vel=25.0)


# ---------------------------------------------------------------- passes
def prepare(case, seed):
    if case["kind"] == "train":
        return _prepare_training(case, seed)
    mesh, arrays = _mesh(case)
    c = _parameters(case)
    s = Solver(mesh, c, precision=case["precision"])
    start = torch.empty((mesh.n_elem, 10), dtype=torch.float64, pin_memory=True)
    start.numpy()[:] = _initial(case, c, arrays["cellCenter"], seed)
    state = dict(case=case, solver=s, start=start, end=torch.empty_like(start, pin_memory=True))
    if case["surrogate"]:
        params, norm = _network(c)
        state["net"] = Surrogate()
        state["net"].set_norm(norm)
        state["net"].set_params(params)
        s.set_surrogate(state["net"], 1e-6, 3)
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        return _run_training(state)
    s = state["solver"]
    watched = []
    s.set_state_async(state["start"].numpy())
    for k in range(case["steps"]):
        if case["stages"]:
            _step_by_stages(s, k, case["dt_every"])
        else:
            s.step()
        if case["monitor"]:
            watched.append(list(s.probe().values()))
    s.get_state_async(state["end"].numpy())
    s.state_join()
    U = state["end"]
    out = {"alpha": U[:, 0], "mass": U[:, 1:3], "momentum": U[:, 3:6], "phase_energy": U[:, 6:8], "energy": U[:, 8],
           "vapour": U[:, 9]}
    if case["monitor"]:
        out["watched"] = np.array(watched).T.copy()
    return out


def _step_by_stages(s, k, dt_every):
    """One step as the reference's explicitLoop writes it."""
    for irk in range(3):
        new_dt = irk == 0 and k % dt_every == 0
        s.compute_rhs(want_signal=new_dt)
        if new_dt:
            s.compute_time_step()
        if irk == 0:
            s.init_rk()
        s.update(irk)
    if s.case.relaxFlag == 0:
        s.relaxation()


def _work_per_step(case):
    """Bytes and operations of a step: per stage the state read and written, the stage-0 state read
    in two of three stages and written in one, each face's vector area, centre and two cells, each
    cell's centre and volume; the relaxation works on the state of the last stage."""
    faces = {"tgv": 6, "mixture": 6, "sod": 4, "bubble": 4, "jet": 4.5, "elements": 5.3}[case["problem"]] / 2
    word = 8 if case["precision"] == "fp64" else 4
    per_stage = 80 + 80 + 80 + faces * (6 * word + 8) + 4 * word
    relaxation = {"sod": 0, "bubble": 6000, "mixture": 6000}.get(case["problem"], 1500)
    return 3 * per_stage, 3 * (650 * faces + 900) + relaxation


def _cells(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return {"sod": 6 * nx * ny * nz, "bubble": 5.29 * nx ** 3, "jet": 3.83 * nx * nx * nz,
            "elements": 2.1 * nx * ny * nz}.get(case["problem"], nx * ny * nz)


def work(case):
    if case["kind"] == "train":
        n = case["samples"] // case["batch"] * case["batch"] + case["batch"]
        return {"bytes": 28.0 * n + 8 * 4 * 8836.0, "flops": 6.0 * 8640 * n}
    b, f = _work_per_step(case)
    n = _cells(case)
    return {"bytes": n * (b * case["steps"] + 160.0), "flops": n * f * case["steps"]}


# ---------------------------------------------------------------- the surrogate
_networks: dict = {}


def _network(c):
    """Trained network of the liquid / vapour mixture (a file that a program loads): parameters and
    normalisation, from equilibrium states that the restatement below solves."""
    key = tuple(c.gamma) + tuple(c.pInf)
    if key not in _networks:
        X, Y = [], []
        g = (np.stack(np.meshgrid(*[np.arange(24)] * 3, indexing="ij"), -1).reshape(-1, 3) + 0.5) * 1e-3
        for seed in range(24):
            U = torch.tensor(physics.perturbed_two_phase_ic(c, g, seed=1000 + seed, vel=25.0).T.copy(), device=DEVICE)
            for _ in range(2):
                V, chemical = _relax(c, U)
                rho = U[1] + U[2]
                e = (U[8] - 0.5 * (U[3:6] ** 2).sum(0) / rho) / rho
                W = _primitive(c, V)
                T = (W[6] + c.pInf[0]) / (c.Cp[0] / c.gamma[0] * (c.gamma[0] - 1) * W[1])
                X.append(torch.stack([rho, e, U[2] / rho], 1)[chemical])
                Y.append(torch.stack([W[6], T, W[0], V[9] / rho], 1)[chemical])
                U = V
        X, Y = torch.cat(X), torch.cat(Y)
        xm, xs, ym, ys = X.mean(0), X.std(0, False), Y.mean(0), Y.std(0, False)
        Z, Q = ((X - xm) / xs).float(), ((Y - ym) / ys).float()
        inverse = torch.linalg.inv(Z.double().T @ Z.double() / len(Z)).float()
        far = torch.einsum("na,ab,nb->n", Z, inverse, Z).max()
        norm = torch.cat([xm.float(), xs.float(), ym.float(), ys.float(), Z.min(0)[0], Z.max(0)[0], inverse.reshape(-1),
                          far.reshape(1)])
        P = [torch.tensor(p, device=DEVICE, requires_grad=True) for p in _layers(np.random.default_rng(3))]
        opt = torch.optim.Adam(P, lr=4e-3)
        steps = 600
        for k in range(steps):
            opt.param_groups[0]["lr"] = 2e-3 * (1 + math.cos(math.pi * k / steps))
            opt.zero_grad()
            torch.nn.functional.mse_loss(_forward(P, Z), Q).backward()
            opt.step()
        _networks[key] = (torch.cat([p.detach().reshape(-1) for p in P]).cpu().numpy(), norm.cpu().numpy())
    return _networks[key]


def _layers(rng):
    out = []
    for k, n in ((3, 64), (64, 64), (64, 64), (64, 4)):
        out += [(rng.standard_normal((k, n)) * math.sqrt(2.0 / k)).astype(np.float32), np.zeros(n, np.float32)]
    return out


def _forward(P, Z):
    for k in range(0, 8, 2):
        Z = Z @ P[k] + P[k + 1]
        if k < 6:
            Z = torch.nn.functional.gelu(Z, approximate="tanh")
    return Z


def _samples(case, seed):
    """Smooth synthetic equilibrium samples (rho, e, Y) -> (p, T, alpha, Y_eq) of the mixture's ranges."""
    rng = np.random.default_rng(seed)
    z = rng.standard_normal((case["samples"], 3)).astype(np.float32)
    k = rng.standard_normal((3, 4)).astype(np.float32)
    y = np.tanh(z @ k) + 0.3 * np.sin(2 * z @ k[:, ::-1])
    scale = np.array([250.0, 1e4, 0.2], np.float32), np.array([3e5, 3.0, 0.25, 0.1], np.float32)
    return (z * scale[0] + np.array([600.0, -9e4, 0.3], np.float32),
            (y * scale[1] + np.array([9e5, 115.0, 0.5, 0.3], np.float32)).astype(np.float32))


def _prepare_training(case, seed):
    X, Y = _samples(case, seed)
    g = Surrogate()
    g.set_data(X, Y)
    g.set_params(np.concatenate([p.reshape(-1) for p in _layers(np.random.default_rng(seed))]))
    n = case["batch"]
    return dict(case=case, net=g, Xs=_standard(X)[:n], Ys=_standard(Y)[:n])


def _standard(A):
    B = A.astype(np.float64)
    return ((B - B.mean(0)) / B.std(0)).astype(np.float32)


def _run_training(state):
    g = state["net"]
    loss, gradient = g.loss_grad(state["Xs"], state["Ys"])
    last = g.train(1, batch=state["case"]["batch"], lr=1e-3, seed=1)
    return {"loss": loss, "gradient": gradient, "last_loss": last, "params": g.params()}


def _exact_training(case, seed):
    X, Y = (torch.tensor(_standard(a)[:case["batch"]], dtype=torch.float64) for a in _samples(case, seed))
    P = [torch.tensor(p, dtype=torch.float64, requires_grad=True) for p in _layers(np.random.default_rng(seed))]
    loss = torch.nn.functional.mse_loss(_forward(P, X), Y)
    loss.backward()
    # the order of an epoch's batches is the framework's own
    return {"loss": float(loss.detach()), "gradient": torch.cat([p.grad.reshape(-1) for p in P]), "last_loss": None,
            "params": None}


# ---------------------------------------------------------------- what the answers are, in 64 bits
def tolerance(case):
    """About four times what two builds that round differently (contracted multiply-adds or not) were
    seen to differ by.  The reference's Newton stops at absolute tolerances, so a change of rounding
    moves the vortex (p about 70) more than the mixture (p about 1e6); the collapsing bubble
    amplifies rounding in its momentum, which starts near rest."""
    if case["kind"] == "train":
        return {"rel": 1e-5, "max": 1e-4}
    mixed = {"tgv": (2e-5, 4e-4), "sod": (2e-5, 4e-4), "bubble": (1.5e-4, 2e-3)}
    fp64 = {"tgv": (4e-8, 1e-6), "bubble": (2e-6, 4e-5)}
    table, rest = (mixed, (2e-6, 2e-4)) if case["precision"] == "mixed" else (fp64, (1e-8, 1e-6))
    rel, largest = table.get(case["problem"], rest)
    return {"rel": max(rel, 2e-6) if case["surrogate"] else rel, "max": largest}


def exact(case, seed):
    if case["kind"] == "train":
        return _exact_training(case, seed)
    _, arrays = _mesh(case)
    c = _parameters(case)
    m = _Faces(arrays)
    U = torch.tensor(_initial(case, c, arrays["cellCenter"], seed).T.copy(), device=DEVICE)
    watched, dt = [], None
    for k in range(case["steps"]):
        U0 = U
        for irk in range(3):
            R, signal = _residual(c, m, U)
            if irk == 0 and k % case["dt_every"] == 0:
                dt = min(c.cfl * float((m.vol ** 0.3333 / signal).min()), c.maxDt)
            a = (0.0, 0.75, 1.0 / 3.0)[irk]
            U = a * U0 + (1 - a) * (U + dt / m.vol * R)
        if c.relaxFlag == 0:
            U, _ = _relax(c, U)
        if case["monitor"]:
            W = _primitive(c, U)
            p = W[0] * W[6] + (1 - W[0]) * W[7]
            watched.append([float(((1 - U[0]) * m.vol).sum()), float(p.max()), float(p.min()),
                            float((W[3:6] ** 2).sum(0).max().sqrt())])
    U = U.T.cpu()
    out = {"alpha": U[:, 0], "mass": U[:, 1:3], "momentum": U[:, 3:6], "phase_energy": U[:, 6:8], "energy": U[:, 8],
           "vapour": U[:, 9]}
    if case["monitor"]:
        out["watched"] = np.array(watched).T.copy()
    return out


class _Faces:
    """Faces of a mesh on the GPU: interior ones (two cells), then boundary ones (one cell, a code)."""

    def __init__(self, a):
        t = lambda x: torch.tensor(np.ascontiguousarray(x), device=DEVICE)   # noqa: E731
        bc = a["boundCond"]
        order = np.argsort(bc != 0, kind="stable")
        self.inner = int((bc == 0).sum())
        self.o = t(a["fc2el"][order, 0].astype(np.int64))
        self.nb = t(a["fc2el"][order, 1].astype(np.int64))[:self.inner]
        self.code = t(bc[order].astype(np.int64))[self.inner:]
        self.n, self.A, self.vol = t(a["n"][order].T), t(a["area"][order]), t(a["volume"])
        self.cells = len(a["volume"])
        x = t(a["cellCenter"].T)
        f = t(a["fcCenter"][order].T)
        self.dO = f - x[:, self.o]
        self.dN = (f + t(a["nbShift"][order].T))[:, :self.inner] - x[:, self.nb]
        mean = self.vol[self.o].clone()
        mean[:self.inner] = 0.5 * (mean[:self.inner] + self.vol[self.nb])
        self.ls2 = (0.325 * mean ** 0.3333333333333) ** 2

    def collect(self, owner, neighbour):
        """Sum of a face quantity over each cell's faces."""
        out = torch.zeros(self.cells, dtype=torch.float64, device=DEVICE)
        return out.index_add_(0, self.o, owner).index_add_(0, self.nb, neighbour)

    def extreme(self, how, start, owner, neighbour):
        out = torch.full((self.cells,), start, dtype=torch.float64, device=DEVICE)
        out.scatter_reduce_(0, self.o, owner, how)
        return out.scatter_reduce_(0, self.nb, neighbour, how)


def _primitive(c, U):
    """[alpha, rho_L, rho_G, u, v, w, p_L, p_G, m_v] of the conserved state (rows)."""
    a = U[0].clamp(c.avfMin / 100, 1 - c.avfMin / 100)
    rl, rg = U[1] / a, U[2] / (1 - a)
    rho = U[1] + U[2]
    p = [(c.gamma[m] - 1) * r * (U[6 + m] / U[1 + m]) - c.gamma[m] * c.pInf[m] - (c.gamma[m] - 1) * c.eta[m] * r
         for m, r in ((0, rl), (1, rg))]
    return torch.stack([a, rl, rg, U[3] / rho, U[4] / rho, U[5] / rho, p[0], p[1], U[9]])


def _ghosts(c, m, s):
    """States beyond the boundary faces of the states `s` on their inner side."""
    n, g, code = m.n[:, m.inner:], s.clone(), m.code
    un = (s[3:6] * n).sum(0)
    slip, wall, inlet = (code == 1) | (code == 4), code == 5, code == 3
    for d in range(3):
        g[3 + d] = torch.where(slip, s[3 + d] - 2 * un * n[d], torch.where(wall, -s[3 + d], s[3 + d]))
    p, T = (c.inletP, c.inletT) if c.inletStateFlag == 1 else (11.4e5, 115.3)
    fixed = {0: 1 - c.avfMin, 1: physics.rho_of_pT(c, 0, p, T), 2: physics.rho_of_pT(c, 1, p, T), 6: p, 7: p, 8: 0.0}
    if c.inletVelFlag == 1:
        fixed.update({3 + d: c.inletVel[d] for d in range(3)})
    for v, x in fixed.items():
        g[v] = torch.where(inlet, torch.full_like(g[v], x), g[v])
    return g


def _sound(c, s, woods):
    c2 = [c.gamma[m] * (s[6 + m] + c.pInf[m]) / s[1 + m] for m in range(2)]
    a, b = s[0], 1 - s[0]
    rho = a * s[1] + b * s[2]
    frozen = torch.sqrt((a * s[1] * c2[0] + b * s[2] * c2[1]) / rho)
    return torch.where(woods, 1 / torch.sqrt(rho * (a / (s[1] * c2[0]) + b / (s[2] * c2[1]))), frozen)


def _energy(c, m, p, rho):
    return (p + c.gamma[m] * c.pInf[m] + (c.gamma[m] - 1) * c.eta[m] * rho) / (rho * (c.gamma[m] - 1))


def _residual(c, m, U):
    """Residual of the conserved state and each cell's largest signal speed."""
    W = _primitive(c, U)
    i, o, nb = m.inner, m.o, m.nb
    beyond = _ghosts(c, m, W[:, o[i:]])
    L, R = torch.empty((9, len(o)), dtype=torch.float64, device=DEVICE), None
    R = torch.empty_like(L)
    grad = torch.empty((9, 3, m.cells), dtype=torch.float64, device=DEVICE)
    for v in range(9):   # Green-Gauss gradient, limited to the face neighbours' range
        w = W[v]
        wo = w[o]
        wn = torch.cat([w[nb], beyond[v]])
        h = 0.5 * (wo + wn) * m.A
        for d in range(3):
            grad[v, d] = m.collect(h * m.n[d], -(h * m.n[d])[:i]) / m.vol
        top = m.extreme("amax", -1e12, wn, wo[:i])
        low = m.extreme("amin", 1e12, wn, wo[:i])

        def share(cell, x):
            own = w[cell]
            diff = own + sum(x[d] * grad[v, d][cell] for d in range(3)) - own
            phi = lambda r: (r * r + r) / (r * r + 1) if c.limiter == 1 else r / 2   # noqa: E731
            f = torch.where(diff > 0, phi((top[cell] - own) / diff), phi((low[cell] - own) / diff))
            return torch.where(diff == 0, torch.ones_like(f), f.clamp(0, 1))

        theta = m.extreme("amin", 1.0, share(o, m.dO), share(nb, m.dN))
        L[v] = wo + theta[o] * sum(m.dO[d] * grad[v, d][o] for d in range(3))
        R[v, :i] = w[nb] + theta[nb] * sum(m.dN[d] * grad[v, d][nb] for d in range(3))
    R[:, i:] = _ghosts(c, m, L[:, i:])
    F, u, p = _hllc(c, m.n, L, R)
    H = F * m.A
    H[3:6] += p * m.A * m.n
    if c.viscFlag == 1:
        _viscous(c, m, W, grad, L, torch.cat([R[:, :i], beyond], 1), H)
    u = u * m.A
    RHS = torch.stack([m.collect(-H[v], H[v, :i]) for v in range(10)])
    su = m.collect(-u, u[:i])
    RHS[0] -= W[0] * su
    RHS[6] += W[0] * W[6] * su
    RHS[7] += (1 - W[0]) * W[7] * su
    pc = W[0] * W[6] + (1 - W[0]) * W[7]
    for d in range(3):
        area = m.A * m.n[d]
        RHS[3 + d] += pc * m.collect(area, -area[:i])

    def signal(s, n):
        return (s[3:6] * n).sum(0).abs() + _sound(c, s, (s[8] > c.chemLimit) & (c.woodsFlag == 1))

    most = signal(L, m.n)
    most[:i] = torch.maximum(most[:i], signal(R[:, :i], m.n[:, :i]))
    return RHS, m.extreme("amax", -1e9, most, most[:i])


def _hllc(c, n, L, R):
    """Advective face flux (10 rows), normal velocity of the face, upwind mixture pressure."""
    uL, uR = (L[3:6] * n).sum(0), (R[3:6] * n).sum(0)
    woods = (0.5 * (L[8] + R[8]) > c.chemLimit) & (c.woodsFlag == 1)
    cL, cR = _sound(c, L, woods), _sound(c, R, woods)
    SL, SR = torch.minimum(uL - cL, uR - cR), torch.maximum(uL + cL, uR + cR)
    pm = [s[0] * s[6] + (1 - s[0]) * s[7] for s in (L, R)]
    rm = [s[0] * s[1] + (1 - s[0]) * s[2] for s in (L, R)]
    Ss = (pm[1] - pm[0] + rm[0] * uL * (SL - uL) - rm[1] * uR * (SR - uR)) / (rm[0] * (SL - uL) - rm[1] * (SR - uR))
    left = (Ss >= 0) | ((c.hllcTieTol > 0) & (Ss.abs() <= c.hllcTieTol * (SL.abs() + SR.abs())))
    s = torch.where(left, L, R)
    un, K = torch.where(left, uL, uR), torch.where(left, SL, SR)
    pm, rho = torch.where(left, *pm), torch.where(left, *rm)
    part = [s[0] * s[1], (1 - s[0]) * s[2]]
    pe = [part[m] * _energy(c, m, s[6 + m], s[1 + m]) for m in range(2)]
    rE = pe[0] + pe[1] + 0.5 * rho * (s[3:6] ** 2).sum(0)
    star = (SL < 0) & (SR >= 0)
    fac = (K - un) / (K - Ss)
    us = s[3:6] + (Ss - un) * n
    spe = []
    for m in range(2):
        r, rs, g = s[1 + m], s[1 + m] * fac, c.gamma[m]
        ps = (s[6 + m] + c.pInf[m]) * ((g - 1) * r - (g + 1) * rs) / ((g - 1) * rs - (g + 1) * r) - c.pInf[m]
        spe.append((s[0] if m == 0 else 1 - s[0]) * rs * _energy(c, m, ps, rs))
    lift = rho if c.hllcEnergyFix == 1 else 1.0
    sE = fac * (rE + lift * (Ss - un) * (Ss + pm / (rho * (K - un))))
    jump = lambda x, y: torch.where(star, K * (x - y), torch.zeros_like(x))   # noqa: E731
    vel = torch.where(star, us, s[3:6])
    u = (vel * n).sum(0)
    rows = [s[0] * u, part[0] * un + jump(part[0] * fac, part[0]), part[1] * un + jump(part[1] * fac, part[1])]
    rows += [rho * s[3 + d] * un + jump(rho * fac * us[d], rho * s[3 + d]) for d in range(3)]
    rows += [torch.where(star, spe[m], pe[m]) * u for m in range(2)]
    rows += [un * (rE + pm) + jump(sE, rE), s[8] * un + jump(s[8] * fac, s[8])]
    return torch.stack(rows), u, pm


def _viscous(c, m, W, grad, L, N, H):
    """Laminar and WALE stresses, and heat conduction, off the face flux H."""
    i, o, nb = m.inner, m.o, m.nb
    mean = lambda q: 0.5 * (q[o] + torch.cat([q[nb], q[o[i:]]]))   # noqa: E731
    g = [[mean(grad[3 + a, d]) for d in range(3)] for a in range(3)]
    nut = 0.0
    if c.turbulence == 1:
        sq = [[sum(g[a][k] * g[k][b] for k in range(3)) for b in range(3)] for a in range(3)]
        tr = sq[0][0] + sq[1][1] + sq[2][2]
        s1 = sum((0.5 * (sq[a][b] + sq[b][a]) - (tr / 3 if a == b else 0.0)) ** 2 for a in range(3) for b in range(3))
        s2 = sum((0.5 * (g[a][b] + g[b][a])) ** 2 for a in range(3) for b in range(3))
        den = s1 ** 1.25 + s2 ** 2.5 + 1e-12
        nut = m.ls2 * torch.where(den < 1e-10, torch.zeros_like(den), s1 ** 1.5) / den
    div = (g[0][0] + g[1][1] + g[2][2]) * (2.0 / 3.0)
    tau = [[g[a][b] + g[b][a] - (div if a == b else 0.0) for b in range(3)] for a in range(3)]
    rho = [s[0] * s[1] + (1 - s[0]) * s[2] for s in (L, N)]
    a = 0.5 * (L[0] + N[0])
    mu = a * c.dynVisc[0] + (1 - a) * c.dynVisc[1] + 0.5 * (rho[0] + rho[1]) * nut
    vel = 0.5 * (L[3:6] + N[3:6])
    for x in range(3):
        H[3 + x] -= mu * m.A * sum(tau[x][d] * m.n[d] for d in range(3))
        H[8] -= mu * m.A * m.n[x] * sum(tau[x][d] * vel[d] for d in range(3))
    if c.heatFlux == 1:
        cv = c.Cp[0] / c.gamma[0] * (c.gamma[0] - 1)
        dT = [(grad[6, d] - (W[6] + c.pInf[0]) / W[1] * grad[1, d]) / (cv * W[1]) for d in range(3)]
        k = mu * (a * c.Cp[0] + (1 - a) * c.Cp[1]) / (a * c.Pr[0] + (1 - a) * c.Pr[1])
        q = sum(mean(dT[d]) * m.n[d] for d in range(3))
        H[8, :i] -= (m.A * k * q)[:i]


def _pressure(c, m, r, e):
    return (c.gamma[m] - 1) * r * e - c.gamma[m] * c.pInf[m] - (c.gamma[m] - 1) * c.eta[m] * r


def _temperature(c, m, r, e):
    return (_pressure(c, m, r, e) + c.pInf[m]) / (c.Cp[m] / c.gamma[m] * (c.gamma[m] - 1) * r)


def _relax(c, U):
    """Relaxed state and the mask of the cells that took the chemical (Gibbs) equilibrium."""
    U = U.clone()
    chemical = torch.zeros(U.shape[1], dtype=torch.bool, device=U.device)
    if c.chemFlag == 1:
        a = U[0].clamp(c.avfMin / 100, 1 - c.avfMin / 100)
        r, e = U[1] / a, U[6] / U[1]
        p, T = _pressure(c, 0, r, e), _temperature(c, 0, r, e)
        chemical = (T > _saturation(c, p, T)) & (a > c.chemLimit)
    for mask, solve in ((~chemical, _thermal), (chemical, _chemical)):
        if bool(mask.any()):
            U[:, mask] = solve(c, U[:, mask])
    return U, chemical


def _saturation(c, P, T):
    cp, cv = c.Cp, [c.Cp[m] / c.gamma[m] for m in range(2)]
    q = cp[1] - cv[1]
    rest = (cp[0] - cp[1] + c.satConst[0] * torch.log10(P) + c.satConst[1]) / q
    rest = rest + (cp[0] - cv[0]) / q * torch.log10(P + c.pInf[0]) - torch.log10(P)
    f = lambda t: rest + (c.eta[0] - c.eta[1]) / q / t + (cp[1] - cp[0]) / q * torch.log10(t)   # noqa: E731
    live = torch.ones_like(T, dtype=torch.bool)
    for _ in range(50):
        if not bool(live.any()):
            break
        fun = f(T)
        T = torch.where(live, T - c.satTempUrf * fun / ((f(T + 1e-3) - fun) / 1e-3), T)
        live = live & (fun.abs() > 1e-2)
    return T


def _newton(U, x, minor, residual, admissible, scale, step, update, limit, enough):
    """Damped Newton with a forward-difference Jacobian on the unknowns `minor` (row indices per
    cell) of x; returns x, with the best admissible iterate where it broke down."""
    best, least = x.clone(), torch.full((x.shape[1],), 1e9, dtype=torch.float32, device=x.device)
    live = torch.arange(x.shape[1], device=x.device)
    k = len(minor)
    for it in range(1, limit + 2):
        if not len(live):
            break
        y = x[:, live]
        at = [row[live] for row in minor]
        y, res = residual(y, live)
        jac = []
        for row in at:
            v = y.gather(0, row[None])[0]
            e = scale(v)
            z, rr = residual(y.scatter(0, row[None], (v + e)[None]), live)
            jac.append((rr - res) / e)
        J = torch.stack(jac, 1).permute(2, 0, 1)
        bad = torch.isnan(J).any(2).any(1) | (torch.linalg.det(J) == 0)
        J[bad] = torch.eye(k, dtype=J.dtype, device=J.device)
        size = res.square().sum(0).sqrt().float()
        better = ~bad & admissible(y) & (size < least[live])
        least[live] = torch.where(better, size, least[live])
        best[:, live] = torch.where(better, y, best[:, live])
        dx = torch.linalg.solve(J, res.T)
        out = bad.clone()
        for q, row in enumerate(at):
            v = y.gather(0, row[None])[0]
            v, wrong = update(row, v, v - step * dx[:, q], dx[:, q], y, live)
            y = y.scatter(0, row[None], v[None])
            out |= wrong
        out |= it > limit
        x[:, live] = torch.where(out, best[:, live], y)
        done = ~(res.abs() > enough).any(0)
        live = live[~(out | done)]
    return x


def _thermal(c, U):
    """Pressure and temperature equilibrium at constant phase masses."""
    lo = c.avfMin / 100
    a = U[0].clamp(lo, 1 - lo)
    part = torch.stack([U[1], U[2]])
    e = torch.stack([U[6], U[7]]) / part
    rho = part.sum(0)
    x = torch.cat([torch.stack([U[1] / a, U[2] / (1 - a)]), e])
    pm = (1 - a > a).long()
    mm = 1 - pm
    e = e + (U[8] - U[6] - U[7]) / rho - 0.5 * (U[3:6] ** 2).sum(0) / rho ** 2

    def close(y, at):
        pick = lambda t, row: t.gather(0, row[None])[0]   # noqa: E731
        P, M, ar, en = pm[at], mm[at], part[:, at], e[:, at]
        s1 = pick(ar, M) / pick(y, M)
        s2 = pick(ar, M) * (pick(y, 2 + M) - pick(en, M))
        y = y.scatter(0, P[None], (pick(ar, P) / (1 - s1))[None])
        return y.scatter(0, (2 + P)[None], (pick(en, P) - s2 / pick(ar, P))[None])

    def residual(y, at):
        y = close(y, at)
        return y, torch.stack([f(c, 0, y[0], y[2]) - f(c, 1, y[1], y[3]) for f in (_pressure, _temperature)])

    x = _newton(U, x, [mm, mm + 2], residual, lambda y: (y[0] > 0) & (y[1] > 0), lambda v: 1e-4 * v, c.thermUrf,
                lambda row, old, new, dx, y, at: (new, torch.zeros_like(new, dtype=torch.bool)), c.thermItrMax, 1e-2)
    x = close(x, torch.arange(x.shape[1], device=x.device))
    V = U.clone()
    V[0] = (part[0] / x[0]).clamp(lo, 1 - lo)
    V[6], V[7] = part[0] * x[2], part[1] * x[3]
    return V


def _chemical(c, U):
    """Pressure, temperature and Gibbs equilibrium at constant mixture mass and energy."""
    lo = c.avfMin / 100
    a = U[0].clamp(lo, 1 - lo)
    rho = U[1] + U[2]
    energy = U[8] - 0.5 * (U[3:6] ** 2).sum(0) / rho
    x = torch.stack([a, 1 - a, U[1] / a, U[2] / (1 - a), U[6] / U[1], U[7] / U[2]])
    pm = (1 - a > a).long()
    mm = 1 - pm

    def gibbs(m, p, T):
        s = c.Cp[m] / c.gamma[m] * torch.log10(T ** c.gamma[m] / (p + c.pInf[m]) ** (c.gamma[m] - 1))
        return c.Cp[m] * T + c.eta[m] - T * (s + (c.satConst[0] * torch.log10(p) + c.satConst[1] if m == 1 else 0.0))

    def close(y, at):
        pick = lambda row: y.gather(0, row[None])[0]   # noqa: E731
        P, M = pm[at], mm[at]
        s1 = pick(M)
        s2 = s1 * pick(M + 2)
        s3 = s2 * pick(M + 4)
        share = 1 - s1
        part = rho[at] - s2
        for row, v in ((P, share), (P + 2, part / share), (P + 4, (energy[at] - s3) / part)):
            y = y.scatter(0, row[None], v[None])
        return y

    def residual(y, at):
        y = close(y, at)
        p = [_pressure(c, m, y[2 + m], y[4 + m]) for m in range(2)]
        T = [_temperature(c, m, y[2 + m], y[4 + m]) for m in range(2)]
        return y, torch.stack([p[0] - p[1], T[0] - T[1], gibbs(0, p[0], T[0]) - gibbs(1, p[1], T[1])])

    def update(row, old, new, dx, y, at):
        """Halve a step that leaves the unknown's range."""
        urf = torch.full_like(new, c.chemUrf)
        share = y.gather(0, (row % 2)[None])[0]
        for kind, over, until in (
                (0, lambda v: v < 0, lambda v: v < c.chemLimit), (0, lambda v: v > 1, lambda v: v > 1 - c.chemLimit),
                (1, lambda v: v < 0, lambda v: v < 0),
                (1, lambda v: share * v > rho[at], lambda v: share * v > rho[at])):
            out = (row // 2 == kind) & over(new)
            for _ in range(12):
                again = out & until(new) & (urf > 0.0005)
                urf = torch.where(again, urf / 2, urf)
                new = torch.where(again, old - urf * dx, new)
        wrong = ((row < 2) & ((new < 0) | (new > 1))) | ((row // 2 == 1) & ((new < 0) | (share * new > rho[at])))
        return new, wrong

    inside = lambda y: (y[0] > 0) & (y[0] < 1) & (y[1] > 0) & (y[1] < 1) & (y[2] > 0) & (y[3] > 0)   # noqa: E731
    x = _newton(U, x, [mm, mm + 2, mm + 4], residual, inside,
                lambda v: torch.where(v.abs() < 1e-9, torch.full_like(v, 1e-10), 1e-5 * v), c.chemUrf, update,
                c.chemItrMax, 1e-1)
    x = close(x, torch.arange(x.shape[1], device=x.device))
    V = U.clone()
    V[0] = x[0].clamp(lo, 1 - lo)
    V[1], V[2] = x[0] * x[2], x[1] * x[3]
    V[6], V[7] = V[1] * x[4], V[2] * x[5]
    V[9] = V[2]
    return V
