"""Performance cases: the calls that programs built on this library make.

The public API works on host arrays (a Loci code hands over its stores), so a
pass takes host data through the whole call: set the state, run the rule or
the steps, read the result back.  A program makes its solver once and runs
many states through it; ``prepare`` therefore keeps the solver of the case it
was last asked for (its mesh does not depend on the seed) and makes the seed's
inputs, in pinned host memory, as the benchmark does.

Sizes and options are those of the workloads in ``flowpsi_b200.cases``, the
benchmark and the tests: split-tet Taylor-Green and farfield boxes up to 128^3
hexes (12.6 M cells), hex cubes and ducts, prisms, the oblique shock, the
flat-plate block with line SGS and Spalart-Allmaras, BDF2 with the
low-dissipation fluxes, the learned start and its training, and the batched
face functions.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from flowpsi_b200 import (FlowPsi, GeneratedMesh, bc, default_params, inviscid_riemann_flux,
                          roe_jacobian)
from flowpsi_b200.learned import LearnedStart

RT = 8314.4621 / 28.96
GAMMA = 1.4
T0, P0 = 300.0, 1e5
A0 = math.sqrt(GAMMA * RT * T0)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(path, mesh="kuhn", n=(16, 16, 16), bcs="periodic", flux="roe",
          limiter="venkatakrishnan", precision="mixed", solver="sgs", sweeps=8, viscous=0, sa=False,
          steps=1, **kw):
    c = {"path": path, "mesh": mesh, "nx": n[0], "ny": n[1], "nz": n[2], "bcs": bcs, "flux": flux,
         "limiter": limiter, "precision": precision, "solver": solver, "sweeps": sweeps,
         "viscous": viscous, "sa": sa, "steps": steps}
    c.update(kw)
    return c


def listed():
    return [
        # one coupling call of a host code with a patch of faces: the fluxes
        # and both Jacobians of a batch (launch and copy latency)
        {"name": "face_batch", "path": "faces", "flux": "hllc", "n": 2000},
        # a host code that drives the rules itself asks for the residual store
        # of a mid-size grid, its norms and the local time step
        _case("residual", n=(40, 40, 40), precision="ref", name="residual_tets40"),
        # the CPU-size steady run of the tests: 32^3 hexes, reference
        # precision, 5 sweeps, 20 steps (launch bound)
        _case("run", "hex", (32, 32, 32), "farfield", precision="ref", sweeps=5, steps=20,
              name="run_hex32_ref"),
        # a small production-precision run, odd sizes
        _case("run", n=(17, 15, 13), bcs="farfield", steps=10, name="run_tets15_mixed"),
        # an ordinary steady run: 1.6 M tets
        _case("run", n=(64, 64, 64), bcs="farfield", steps=5, name="run_tets64_mixed"),
        # the benchmark's grid, the largest: 12.6 M tets
        _case("run", n=(128, 128, 128), steps=5, name="run_tets128_mixed"),
        # supersonic hexes, HLLE + Barth, odd sizes
        _case("run", "hex", (95, 81, 77), "shock", flux="hlle", limiter="barth", steps=4,
              name="run_shock_hex"),
        # the boundary layer: line SGS over the wall-normal columns, SA
        _case("run", "bl", (128, 64, 32), "wall", solver="lsgs", viscous=2, sa=True, steps=4,
              name="run_boundary_layer_sa"),
        # time-accurate vortex with the low-dissipation flux, viscous, FP64:
        # explicit blocks; two BDF2 steps of three Newton iterations
        _case("time_step", n=(28, 28, 28), flux="kec", precision="fp64", viscous=1, sweeps=5,
              steps=2, name="bdf2_kec_tets28_fp64"),
        # a linear system solved to a tolerance, as training sets are made
        _case("tolerance", n=(48, 48, 48), precision="ref", name="solve_to_tol_tets48"),
        # steps from the learned start with the rejection rule
        _case("learned_step", n=(48, 48, 48), bcs="farfield", steps=3, name="learned_step_tets48"),
        # one training pass over a snapshot of the size that the training
        # set's regions have (196,608 cells)
        _case("train", n=(32, 32, 32), precision="ref", name="train_pass_197k"),
    ]


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def box(a, b):  # three sizes near one another, odd ones among them
        m = logint(a, b)
        return tuple(max(a, min(b, m + rng.randint(-(m // 8) - 1, m // 8 + 1))) for _ in range(3))

    path = rng.choice(["faces", "residual", "run", "run", "run", "run_bl", "time_step",
                       "tolerance", "learned_step", "train"])
    prec = rng.choice(["mixed", "mixed", "ref", "fp64"])
    if path == "faces":
        return {"path": path, "flux": rng.choice(["hllc", "roe", "hlle"]), "n": logint(300, 1000000)}
    if path == "run_bl":
        solver = rng.choice(["lsgs", "lsgs", "sgs"])
        viscous = rng.choice([1, 2, 2])
        return _case("run", "bl", (logint(24, 160), logint(16, 72), logint(8, 40)), "wall",
                     precision=prec, solver=solver, viscous=viscous,
                     sa=viscous == 2 and rng.random() < 0.7, steps=rng.randint(3, 6))
    if path == "time_step":
        return _case(path, n=box(8, 40), flux=rng.choice(["kec", "ssf", "roe", "hllc"]),
                     precision=prec, viscous=rng.choice([0, 1]), sweeps=rng.randint(3, 8),
                     steps=rng.randint(1, 2))
    if path in ("tolerance", "train"):
        return _case(path, n=box(8, 40), precision=prec)
    if path == "learned_step":
        return _case(path, n=box(8, 56), bcs="farfield", precision=prec, steps=rng.randint(2, 4))
    mesh = rng.choice(["kuhn", "kuhn", "hex", "prism"])
    bcs = rng.choice(["periodic", "farfield", "duct"] if mesh != "hex" else
                     ["periodic", "farfield", "duct", "shock"])
    flux = "hlle" if bcs == "shock" else rng.choice(["roe", "roe", "hllc", "hlle"])
    limiter = "barth" if bcs == "shock" else rng.choice(["venkatakrishnan", "venkatakrishnan",
                                                         "barth"])
    top = {"kuhn": 72, "hex": 110, "prism": 90}[mesh]
    return _case(path, mesh, box(8, top), bcs, flux=flux, limiter=limiter, precision=prec,
                 sweeps=rng.randint(4, 8), steps=1 if path == "residual" else rng.randint(4, 10))


# ---------------------------------------------------------------------------
# meshes, options and states
# ---------------------------------------------------------------------------
def _box(case):
    """side lengths of the case's box"""
    if case["mesh"] == "bl":
        return (1.0, 1.0, 0.25)
    s = 2.0 * math.pi if case["bcs"] in ("periodic", "farfield") and case["mesh"] == "kuhn" else 1.0
    m = max(case["nx"], case["ny"], case["nz"])
    return tuple(s * case[k] / m for k in ("nx", "ny", "nz"))


def _freestream(case):
    """(T, p, u) of the case's undisturbed flow"""
    M = {"periodic": 0.1, "farfield": 0.5, "duct": 0.5, "shock": 2.0, "wall": 0.3}[case["bcs"]]
    p = P0
    if case["viscous"] and case["bcs"] == "wall":  # Re = 1e6 per unit length
        p = 1e6 * (1.458e-6 * T0 ** 1.5 / (T0 + 110.4)) / (M * A0) * RT * T0
    return T0, p, M * A0


def _mesh(case):
    n, L, kind = (case["nx"], case["ny"], case["nz"]), _box(case), case["mesh"]
    T, p, U = _freestream(case)
    jitter = 0.1 if kind == "kuhn" else 0.0
    ff = bc("farfield", T=T, pg=p, u=(U, 0.0, 0.0))
    if case["bcs"] == "periodic":
        return GeneratedMesh(kind, n=n, L=L, jitter=jitter)
    if case["bcs"] == "farfield":
        return GeneratedMesh(kind, n=n, L=L, jitter=jitter, bc_side=(0,) * 6, bcs=[ff])
    if case["bcs"] == "duct":  # total conditions in, mean back pressure out
        f = 1.0 + 0.2 * 0.25
        ins = bc("isentropicInflow", T=T * f, pg=p * f ** 3.5)
        out = bc("outflowMean", T=T, pg=1.02 * p)
        return GeneratedMesh(kind, n=n, L=L, jitter=jitter, bc_side=(0, 1, -1, -1, -1, -1),
                             bcs=[ins, out])
    if case["bcs"] == "shock":
        return GeneratedMesh(kind, n=n, L=L, bc_side=(0, 1, 1, 1, 1, 1),
                             bcs=[bc("supersonicInflow", T=T, pg=p, u=(U, 0.0, 0.0)),
                                  bc("supersonicOutflow", T=T, pg=p, u=(U, 0.0, 0.0))])
    ffw = bc("farfield", T=T, pg=p, u=(U, 0.0, 0.0), nu_t=_nut(case) if case["sa"] else 0.0)
    wall = bc("viscousWall" if case["viscous"] else "reflecting", T=T, pg=p)
    return GeneratedMesh("bl", n=n, L=L, dy0=1e-6, growth=1.15, bc_side=(0, 0, 1, 0, -1, -1),
                         bcs=[ffw, wall])


def _nut(case):
    T, p, _ = _freestream(case)
    return 3.0 * (1.458e-6 * T ** 1.5 / (T + 110.4)) / (p / (RT * T))


def _params(case):
    kw = dict(flux=case["flux"], limiter=case["limiter"], solver=case["solver"],
              gauss_seidel_iter=case["sweeps"], cflmax=50.0, precision=case["precision"],
              viscous=case["viscous"], turbulence=1 if case["sa"] else 0)
    if case["path"] == "time_step":
        h = min(_box(case)) / case["nx"]
        kw.update(time_accurate=1, newton_iters=3, cflmax=0.0, dtmax=0.2 * h / A0)
    return default_params(**kw)


class _Kept:
    """The solver of one case: what a program makes once."""

    def __init__(self, case):
        self.mesh = _mesh(case)
        self.solver = FlowPsi(self.mesh, _params(case))
        if case["solver"] == "lsgs":
            self.solver.set_lines(self.mesh.lines_along(1))
        T, p, U = _freestream(case)
        if case["viscous"] == 2 and not case["sa"]:
            chi3 = 3.0 ** 3
            self.solver.set_eddy_viscosity(np.full(self.solver.ncells, _nut(case) * (p / (RT * T))
                                                   * chi3 / (chi3 + 7.1 ** 3)))
        cc = torch.from_numpy(self.solver.geometry()["cellcenter"]).cuda()
        self.state = _base_state(case, cc)


def _base_state(case, cc):
    """(T, p, u[nc,3]) on the GPU before the seed's noise"""
    T, p, U = _freestream(case)
    nc = cc.shape[0]
    one = torch.ones(nc, dtype=torch.float64, device=cc.device)
    u = torch.zeros(nc, 3, dtype=torch.float64, device=cc.device)
    if case["bcs"] == "periodic":  # Taylor-Green vortex
        L = _box(case)
        x, y, z = (cc[:, k] * (2.0 * math.pi / L[k]) for k in range(3))
        u[:, 0] = U * torch.sin(x) * torch.cos(y) * torch.cos(z)
        u[:, 1] = -U * torch.cos(x) * torch.sin(y) * torch.cos(z)
        rho = p / (RT * T)
        pp = p + rho * U * U / 16.0 * (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0)
        return pp / (rho * RT), pp, u
    u[:, 0] = U
    if case["bcs"] != "shock":
        return T * one, p * one, u
    # Rankine-Hugoniot jump across a plane tilted 30 degrees
    n = torch.tensor([math.cos(math.pi / 6), math.sin(math.pi / 6), 0.0], dtype=torch.float64,
                     device=cc.device)
    mid = torch.tensor(_box(case), dtype=torch.float64, device=cc.device) / 2
    mn2 = (2.0 * math.cos(math.pi / 6)) ** 2
    p2 = p * (1 + 2 * GAMMA / (GAMMA + 1) * (mn2 - 1))
    rr = (GAMMA + 1) * mn2 / ((GAMMA - 1) * mn2 + 2)
    down = (cc - mid) @ n > 0
    un = U * math.cos(math.pi / 6)
    u = torch.where(down[:, None], u + (un / rr - un) * n, u)
    return torch.where(down, T * p2 / p / rr, T * one), torch.where(down, p2 * one, p * one), u


_kept = {}  # the one solver kept between preparations, by the options it was made with


def _keep(case):
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if key not in _kept:
        _kept.clear()
        _kept[key] = _Kept(case)
    return _kept[key]


def _pinned(t):
    """a tensor's values in pinned host memory, as a numpy array"""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _noisy(case, base, seed):
    """the seed's state in pinned host memory: 1% noise in T, p and u"""
    T, p, u = base
    g = torch.Generator(device=T.device).manual_seed(seed)
    umax = u.abs().max()

    def r(x):
        return torch.randn(x.shape, generator=g, dtype=x.dtype, device=x.device)

    return _pinned(T * (1 + 0.01 * r(T))), _pinned(p * (1 + 0.01 * r(p))), \
        _pinned((u + 0.01 * umax * r(u)).reshape(-1))


def _faces(case, seed):
    """face states [pg,T,u,v,w] of neighbouring cells, unit normals, areas"""
    r = np.random.default_rng(seed)
    n = case["n"]
    q = np.stack([P0 * r.uniform(0.8, 1.2, n), T0 * r.uniform(0.8, 1.2, n),
                  *(A0 * r.uniform(-1.5, 1.5, (3, n)))], 1)
    q2 = q * (1 + 0.05 * r.standard_normal((n, 5)))
    an = r.standard_normal((n, 3))
    an /= np.linalg.norm(an, axis=1)[:, None]
    return q, q2, an, r.uniform(0.5, 1.5, n) * 1e-3


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["path"] == "faces":
        return {"case": case, "faces": _faces(case, seed)}
    kept = _keep(case)
    s = kept.solver
    st = {"case": case, "solver": s, "kept": kept, "state": _noisy(case, kept.state, seed)}
    st["out"] = tuple(_pinned(torch.empty(a.shape, dtype=torch.float64)) for a in st["state"])
    if case["sa"]:
        r = np.random.default_rng(seed)
        st["nut"] = _nut(case) * (1 + 0.1 * r.random(s.ncells))
    if case["path"] in ("learned_step", "train"):
        # a model with weights as training leaves them: a small non-zero head
        m = LearnedStart(seed=1)
        w = m.get_params()
        head = 5 * 64 + 5
        scale = 0.02 if case["path"] == "learned_step" else 0.2
        w[-head:] = scale * np.random.default_rng(3).standard_normal(head).astype(np.float32)
        m.set_params(w)
        st["model"] = m
    if case["path"] == "train":
        s.set_state(*st["state"])
        s.residual(want_src=False)
        s.assemble()
        s.sweeps(10)
        dq = s.get_iterate()
        s.assemble()
        st["model"].add_snapshot(s, dq)
    return st


def _norms(hist):
    keys = ("rtrms", "etrms", "mtrms", "rtmax", "etmax", "mtmax")
    return np.array([[h[k] for k in keys] for h in hist])


def run(st):
    case, path = st["case"], st["case"]["path"]
    if path == "faces":
        qL, qR, an, area = st["faces"]
        return {"flux": inviscid_riemann_flux(case["flux"], qL, qR, an, area),
                "fjp": roe_jacobian(qL, qR, an, area, 1), "fjm": roe_jacobian(qL, qR, an, area, -1)}
    if path == "train":
        loss, grad = st["model"].loss_grad(0)
        return {"loss": loss, "grad": grad}
    s = st["solver"]
    s.set_state(*st["state"])
    if path == "residual":
        src, norms = s.residual()
        return {"src": src, "norms": _norms([norms]), "dtau": s.dtau()}
    if path == "tolerance":
        s.residual(want_src=False)
        s.assemble()
        n = s.sweeps_to_tolerance(1e-2, 40)
        return {"sweeps": n, "dq": s.get_iterate()}
    if case["sa"]:
        s.set_nutilde(st["nut"])
    if path == "time_step":
        hist = [h for _ in range(case["steps"]) for h in s.time_step()]
    elif path == "learned_step":
        hist = [s.newton_step_ex("learned", st["model"])["after"] for _ in range(case["steps"])]
    else:
        hist = s.run(case["steps"])
    T, p, u = s.get_state(out=st["out"])
    out = {"T": T, "p": p, "u": u, "norms": _norms(hist)}
    if case["sa"]:
        out["nut"] = s.nutilde()
    return out


# ---------------------------------------------------------------------------
# the work a pass cannot do without
# ---------------------------------------------------------------------------
def _counts(case):
    """cells, interior faces (boundary faces are left out)"""
    h = case["nx"] * case["ny"] * case["nz"]
    per = {"hex": (1, 3.0), "bl": (1, 3.0), "prism": (2, 5.0), "kuhn": (6, 12.0)}[case["mesh"]]
    return per[0] * h, per[1] * h


def work(case):
    if case["path"] == "faces":
        # both states, normal and area in; the flux (FP64) and two FP32 blocks out
        return {"bytes": case["n"] * (14 * 8 + 5 * 8 + 2 * 100), "flops": case["n"] * 1200}
    nc, nf = _counts(case)
    if case["path"] == "train":
        # features, graph, targets and the FP32 gradient once; the three
        # layers' forward (2 products) and backward (4 products)
        per_cell = 3 * 2 * (64 * 80 + 2 * 64 * 128)
        return {"bytes": nc * (160 + 20 + 16), "flops": nc * per_cell}
    tb = 8 if case["precision"] == "fp64" else 4
    compact = not case["viscous"] and case["solver"] != "lsgs"
    # state in and out; geometry per residual: normal, area, two face vectors,
    # two cell ids per face; volume and least-squares inverse per cell
    resid = nc * (40 + 40 + 56) + nf * 88
    # the system once out and once in per symmetric sweep: LU, B and iterate
    # per cell, a block per face side
    system = nc * 35 * tb + 2 * nf * (15 if compact else 25) * tb
    sweeps = 10 if case["solver"] == "lsgs" else case["sweeps"]
    fl_res = nf * 900 + nc * 400
    fl_sys = nf * 700 + nc * 200
    fl_sweep = 2 * (2 * nf * 60 + nc * 60)
    steps = case["steps"] * (3 if case["path"] == "time_step" else 1)
    if case["path"] == "residual":
        return {"bytes": resid + nc * 8, "flops": fl_res}
    if case["path"] == "tolerance":
        steps, sweeps = 1, 4
    if case["path"] == "learned_step":
        # the network: features in, the start out, three layers
        return {"bytes": steps * (2 * resid + (1 + sweeps) * system + nc * 240),
                "flops": steps * (2 * fl_res + fl_sys + sweeps * fl_sweep + nc * 43000)}
    return {"bytes": steps * (resid + (1 + sweeps) * system),
            "flops": steps * (fl_res + fl_sys + sweeps * fl_sweep)}


# ---------------------------------------------------------------------------
# 64-bit values, written out from the method (numpy and torch only)
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["path"] == "faces":
        qL, qR, an, area = (torch.from_numpy(a) for a in _faces(case, seed))
        # [pg,T,u,v,w] -> [T,u,v,w,pg]
        L, R = (torch.cat([q[:, 1:], q[:, :1]], 1) for q in (qL, qR))
        flux = _FLUX[case["flux"]](L, R, an, area)
        return {"flux": flux.numpy(), "fjp": _roe_block(L, R, an, area, 1.0).numpy(),
                "fjm": _roe_block(L, R, an, area, -1.0).numpy()}
    if case["path"] == "residual" and case["bcs"] == "periodic" and _counts(case)[0] <= 500000:
        return _exact_residual(case, seed)
    # boundary states, truncated relaxations, runs and the BF16 network: none
    return None


def _roe_average(L, R, n):
    rl, rr = L[:, 4] / (RT * L[:, 0]), R[:, 4] / (RT * R[:, 0])
    wl, wr = rl.sqrt(), rr.sqrt()
    w = wl / (wl + wr)

    def mean(a, b):
        return a * w + b * (1 - w)

    u = mean(L[:, 1:4].T, R[:, 1:4].T).T
    cp = GAMMA * RT / (GAMMA - 1)
    h0 = mean(cp * L[:, 0] + 0.5 * (L[:, 1:4] ** 2).sum(1), cp * R[:, 0] + 0.5 * (R[:, 1:4] ** 2).sum(1))
    a = ((GAMMA - 1) * (h0 - 0.5 * (u ** 2).sum(1))).sqrt()
    return wl * wr, u, h0, a, (u * n).sum(1)


def _physical(q, n):
    """conserved variables and flux through n of [T,u,v,w,p]"""
    rho = q[:, 4] / (RT * q[:, 0])
    un = (q[:, 1:4] * n).sum(1)
    e = rho * (RT * q[:, 0] / (GAMMA - 1) + 0.5 * (q[:, 1:4] ** 2).sum(1))
    U = torch.cat([rho[:, None], rho[:, None] * q[:, 1:4], e[:, None]], 1)
    F = U * un[:, None]
    F[:, 1:4] += q[:, 4:5] * n
    F[:, 4] += q[:, 4] * un
    return U, F, un, (GAMMA * RT * q[:, 0]).sqrt()


def _roe_matrix(avg, n, lam):
    """d(conserved)/d(T,u,v,w,p) of the Roe state with the eigenvalues lam =
    (un, un - a, un + a) of the flux Jacobian put in: R diag(lam) R^-1 dU/dq"""
    rho, u, h0, a, un = avg
    N = rho.shape[0]
    l1, l2, l3 = lam
    z = torch.zeros(N, 5, 5, dtype=rho.dtype)
    # a jump in q splits into an entropy/shear part and two acoustic parts with
    # strengths (dp -+ rho a dun) / (2 a^2)
    cp = GAMMA * RT / (GAMMA - 1)
    T = a * a / (GAMMA * RT)
    ek = 0.5 * (u ** 2).sum(1)
    for j in range(5):
        dT = torch.full_like(rho, 1.0 if j == 0 else 0.0)
        du = torch.zeros_like(u)
        if 1 <= j <= 3:
            du[:, j - 1] = 1.0
        dp = torch.full_like(rho, 1.0 if j == 4 else 0.0)
        drho = dp / (RT * T) - rho / T * dT
        dun = (du * n).sum(1)
        am, ap = (dp - rho * a * dun) / (2 * a * a), (dp + rho * a * dun) / (2 * a * a)
        ent = drho - dp / (a * a)
        ut = du - dun[:, None] * n
        z[:, 0, j] = l1 * ent + l2 * am + l3 * ap
        z[:, 1:4, j] = (l1 * ent)[:, None] * u + (l1 * rho)[:, None] * ut \
            + (l2 * am)[:, None] * (u - a[:, None] * n) + (l3 * ap)[:, None] * (u + a[:, None] * n)
        z[:, 4, j] = l1 * (ent * ek + rho * (u * ut).sum(1)) + l2 * am * (h0 - un * a) + l3 * ap * (h0 + un * a)
    return z


def _roe_block(L, R, n, area, d):
    """one side's smoothed Roe Jacobian: l -> (l +- sqrt(l^2 + (0.02 spread)^2)) / 2"""
    avg = _roe_average(L, R, n)
    a, un = avg[3], avg[4]
    e2 = (0.02 * 2 * a) ** 2
    lam = [0.5 * (l + d * (l * l + e2).sqrt()) for l in (un, un - a, un + a)]
    return _roe_matrix(avg, n, lam) * area[:, None, None]


def _roe_flux(L, R, n, area):
    avg = _roe_average(L, R, n)
    rho, u, h0, a, un = avg
    (_, Fl, ul, al), (_, Fr, ur, ar) = _physical(L, n), _physical(R, n)
    lam = [un.abs()]
    for s in (-1.0, 1.0):  # Harten-Hyman fix of the acoustic waves
        l = un + s * a
        w = torch.clamp(torch.maximum(l - (ul + s * al), (ur + s * ar) - l), min=0.0)
        lam.append(torch.where(l.abs() < w, 0.5 * (l * l / w.clamp(min=1e-300) + w), l.abs()))
    d = R - L
    (l1, l2, l3), dun = lam, (d[:, 1:4] * n).sum(1)
    # the scheme's primitive jumps, with rho(T, p) linearised at the Roe state
    T = a * a / (GAMMA * RT)
    drho = d[:, 4] / (RT * T) - rho / T * d[:, 0]
    am, ap = (d[:, 4] - rho * a * dun) / (2 * a * a), (d[:, 4] + rho * a * dun) / (2 * a * a)
    ent, ut = drho - d[:, 4] / (a * a), d[:, 1:4] - dun[:, None] * n
    D = torch.zeros_like(Fl)
    D[:, 0] = l1 * ent + l2 * am + l3 * ap
    D[:, 1:4] = (l1 * ent)[:, None] * u + (l1 * rho)[:, None] * ut + (l2 * am)[:, None] * (u - a[:, None] * n) \
        + (l3 * ap)[:, None] * (u + a[:, None] * n)
    D[:, 4] = l1 * (ent * 0.5 * (u ** 2).sum(1) + rho * (u * ut).sum(1)) + l2 * am * (h0 - un * a) \
        + l3 * ap * (h0 + un * a)
    return 0.5 * (Fl + Fr - D) * area[:, None]


def _waves(L, R, n):
    _, _, _, a, un = _roe_average(L, R, n)
    l, r = _physical(L, n), _physical(R, n)
    return l, r, torch.minimum(un - a, l[2] - l[3]), torch.maximum(un + a, r[2] + r[3])


def _hlle_flux(L, R, n, area):
    (Ul, Fl, _, _), (Ur, Fr, _, _), sl, sr = _waves(L, R, n)
    sl, sr = sl.clamp(max=0.0)[:, None], sr.clamp(min=0.0)[:, None]
    return (sr * Fl - sl * Fr + sl * sr * (Ur - Ul)) / (sr - sl) * area[:, None]


def _hllc_flux(L, R, n, area):
    (Ul, Fl, ul, _), (Ur, Fr, ur, _), sl, sr = _waves(L, R, n)
    rl, rr, pl, pr = Ul[:, 0], Ur[:, 0], L[:, 4], R[:, 4]
    sm = (rr * ur * (sr - ur) - rl * ul * (sl - ul) + pl - pr) / (rr * (sr - ur) - rl * (sl - ul))
    ps = rl * (ul - sl) * (ul - sm) + pl

    def star(U, q, un, s, F):
        V = U * (s - un)[:, None]
        V[:, 1:4] += (ps - q[:, 4])[:, None] * n
        V[:, 4] += ps * sm - q[:, 4] * un
        return F + s[:, None] * (V / (s - sm)[:, None] - U)

    out = torch.where((sm >= 0)[:, None], star(Ul, L, ul, sl, Fl), star(Ur, R, ur, sr, Fr))
    out = torch.where((sl > 0)[:, None], Fl, out)
    return torch.where((sr < 0)[:, None], Fr, out) * area[:, None]


_FLUX = {"roe": _roe_flux, "hllc": _hllc_flux, "hlle": _hlle_flux}


def _exact_geometry(mesh):
    """area vectors, face vectors from both cells and volumes of a periodic
    mesh: faces fanned about their node average, cells from the pyramids"""
    m = mesh.arrays()
    x = torch.from_numpy(np.array(m.xyz)).reshape(-1, 3)
    off, nodes = torch.from_numpy(np.array(m.face_off)), torch.from_numpy(np.array(m.face_nodes)).long()
    cl, cr = (torch.from_numpy(np.array(a)).long() for a in (m.cl, m.cr))
    sh = torch.zeros(m.nfaces, 3, dtype=torch.float64) if m.pshift is None else \
        torch.from_numpy(np.array(m.pshift)).reshape(-1, 3)
    k = off[1:] - off[:-1]
    f = torch.repeat_interleave(torch.arange(m.nfaces), k)
    i = torch.arange(nodes.numel()) - off[f]
    p0, p1 = x[nodes], x[nodes[off[f] + (i + 1) % k[f]]]

    def per_face(v):
        return torch.zeros(m.nfaces, *v.shape[1:], dtype=torch.float64).index_add_(0, f, v)

    xa = per_face(p0) / k[:, None]
    t = 0.5 * torch.linalg.cross(p0 - xa[f], p1 - xa[f])
    w = t.norm(dim=1)
    av = per_face(t)
    fc = per_face(w[:, None] / 3 * (xa[f] + p0 + p1)) / per_face(w)[:, None]
    vol, cc = torch.zeros(m.ncells, dtype=torch.float64), torch.zeros(m.ncells, 3, dtype=torch.float64)
    cnt, xr = torch.zeros(m.ncells, dtype=torch.float64), torch.zeros(m.ncells, 3, dtype=torch.float64)
    for c, s in ((cl, 0.0), (cr, 1.0)):
        xr.index_add_(0, c, fc - s * sh)
        cnt.index_add_(0, c, torch.ones_like(c, dtype=torch.float64))
    xr /= cnt[:, None]
    for c, s, sg in ((cl, 0.0, 1.0), (cr, 1.0, -1.0)):
        o = s * sh[f] + xr[c[f]]
        a, b, d = xa[f] - o, p0 - o, p1 - o
        v = sg * (a * torch.linalg.cross(b, d)).sum(1) / 6
        vol.index_add_(0, c[f], v)
        cc.index_add_(0, c[f], (v * 0.25)[:, None] * (4 * xr[c[f]] + a + b + d))
    cc /= vol[:, None]
    return cl, cr, av, fc - cc[cl], fc - sh - cc[cr], vol


def _exact_residual(case, seed):
    """src, the norms and dtau of the inviscid residual of a periodic mesh"""
    kept = _keep(case)
    T, p, u = (torch.from_numpy(np.array(a)) for a in _noisy(case, kept.state, seed))
    q = torch.cat([T[:, None], u.reshape(-1, 3), p[:, None]], 1)
    cl, cr, av, rl, rr, vol = _exact_geometry(kept.mesh)
    nc = q.shape[0]
    area = av.norm(dim=1)
    n = av / area[:, None]

    def add(vl, vr):
        z = torch.zeros(nc, *vl.shape[1:], dtype=torch.float64)
        return z.index_add_(0, cl, vl).index_add_(0, cr, vr)

    # unweighted least squares over the face neighbours
    d, dq = rl - rr, q[cr] - q[cl]
    dd = d[:, :, None] * d[:, None, :]
    b = d[:, :, None] * dq[:, None, :]
    g = torch.linalg.solve(add(dd, dd), add(b, b))  # [nc, xyz, var]
    hi, lo = q.clone(), q.clone()
    for c, o in ((cl, cr), (cr, cl)):
        idx = c[:, None].expand(-1, 5)
        hi.scatter_reduce_(0, idx, q[o], "amax")
        lo.scatter_reduce_(0, idx, q[o], "amin")
    phi = torch.full((nc, 5), math.inf, dtype=torch.float64)
    eps2 = vol[:, None]  # (Kl V^(1/3))^3, Kl = 1
    for c, r in ((cl, rl), (cr, rr)):
        d2 = torch.einsum("fx,fxv->fv", r, g[c])
        d1 = torch.where(d2 > 0, hi[c] - q[c], lo[c] - q[c])
        if case["limiter"] == "barth":
            y = d1 / torch.where(d2 == 0, torch.ones_like(d2), d2)
        else:
            e = eps2[c]
            y = ((d1 * d1 + e) + 2 * d2 * d1) / (d1 * d1 + 2 * d2 * d2 + d1 * d2 + e)
        y = torch.where(d2 == 0, torch.ones_like(y), y.clamp(max=1.0))
        phi.scatter_reduce_(0, c[:, None].expand(-1, 5), y, "amin")
    ql = q[cl] + phi[cl] * torch.einsum("fx,fxv->fv", rl, g[cl])
    qr = q[cr] + phi[cr] * torch.einsum("fx,fxv->fv", rr, g[cr])
    low = 0.1 * torch.minimum(q[cl], q[cr])
    for v in (0, 4):  # floors of T and p
        ql[:, v] = torch.maximum(ql[:, v], low[:, v])
        qr[:, v] = torch.maximum(qr[:, v], low[:, v])
    F = _FLUX[case["flux"]](ql, qr, n, area)
    src = add(-F, F)
    # spectral radii of the cell-centre states, the CFL and urelax limits
    lam = torch.maximum(*((q[c][:, 1:4] * n).sum(1).abs() + (GAMMA * RT * q[c][:, 0]).sqrt() for c in (cl, cr)))
    dt = (50.0 * vol / (0.5 * add(lam * area, lam * area))).clamp(max=1.0)
    un2 = (q[:, 1:4] ** 2).sum(1)
    rho = q[:, 4] / (RT * q[:, 0])
    srho = src[:, 0]
    se = src[:, 4] - (q[:, 1:4] * src[:, 1:4]).sum(1) + 0.5 * un2 * srho  # change of rho e
    dp = (GAMMA - 1) * se / vol
    dT = q[:, 0] * (dp / q[:, 4] - srho / vol / rho)
    dt = torch.minimum(dt, 0.2 * q[:, 0] / (dT.abs() + 1e-30))
    # the rule bounds the pressure by rho / T times the energy change per volume
    dt = torch.minimum(dt, 0.2 * q[:, 4] / ((rho / q[:, 0] * se / vol).abs() + 1e-30))
    a = src / vol[:, None]
    w = vol / vol.sum()

    def signed_max(v):
        return float(v.reshape(-1)[v.abs().reshape(-1).argmax()])

    norms = [math.sqrt(float((w * a[:, 0] ** 2).sum())), math.sqrt(float((w * a[:, 4] ** 2).sum())),
             math.sqrt(float((w[:, None] * a[:, 1:4] ** 2).sum() / 3)), signed_max(a[:, 0]),
             signed_max(a[:, 4]), signed_max(a[:, 1:4])]
    return {"src": src.numpy(), "norms": np.array([norms]), "dtau": dt.numpy()}
