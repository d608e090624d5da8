"""Performance cases: the work a user of this package has it do, through its
public entry points.

What the cases stand for:

  step   one ``solver.step.step`` call with a prepared plan: halo fill, boundary
         conditions and the three TVD-RK3 stages of every block.  A solver's
         inner loop, from the 32^3 Taylor-Green block (latency and launches
         count) to four curvilinear 128^3 blocks and the 24 uneven blocks with
         farfield faces (26.5 M cells, the largest).
  run    ``solver.run.run``: the monitored time loop (captured steps, residual
         log, state check), for one block and for an ensemble of independent
         instances with their own viscosity and time step.
  grad   ``solver.adjoint.adjoint_kinetic_energy``: the checkpointed forward and
         reverse sweep (the backward direction of the step).
  rhs    ``rhs.invscd.compute_invscd_rhs`` and ``rhs.viscous.compute_viscous_rhs``
         of one block, the calls a program with its own time integrator makes.

Each in FP64 (``precision="f64"``, the drop-in path) and in the FP32-flux /
FP64-state variant (``"f32"``), with both limiters and both viscosity laws.  The
flows, Mach and Reynolds numbers, noise levels and sizes are those of the
package's configurations (``famrdp_jax_b200/cases.py``) and tests; inputs are
drawn on the GPU from the seed.  A case is a dict of plain values.

``exact`` evaluates the same step, loop, gradient or right-hand side in plain
torch FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

GHOST = 2
GAMMA = 1.4
PRANDTL = 0.72
EPS_ENTROPY = 0.1
CFL = 0.5
FARFIELD, WALL, SYMMETRY = "farfield", "wall", "symmetry"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest calls: one step of the 32^3 Taylor-Green block (M 0.1,
        # Re 1600, constant viscosity), both precisions
        dict(name="step_tgv32_f32", do="step", flow="tgv", n=32, M=0.1, Re=1600.0, law="constant",
             limiter="minmod", precision="f32"),
        dict(name="step_tgv32_f64", do="step", flow="tgv", n=32, M=0.1, Re=1600.0, law="constant",
             limiter="minmod", precision="f64"),
        # a monitored FP64 time loop of one ensemble-sized block
        dict(name="run_tgv64_f64", do="run", flow="tgv", n=64, M=0.3, Re=800.0, law="sutherland",
             limiter="minmod", precision="f64", steps=20, every=10),
        # odd extents between walls and symmetry planes, the other limiter
        dict(name="step_duct_f64", do="step", flow="duct", ni=97, nj=61, nk=45, M=0.3, Re=1e4, law="sutherland",
             limiter="vanleer", precision="f64"),
        # both right-hand sides of one ragged block
        dict(name="rhs_ragged_f64", do="rhs", flow="duct", ni=127, nj=66, nk=51, M=0.5, Re=1e4, law="sutherland",
             limiter="minmod", precision="f64"),
        # the headline: four curvilinear 128^3 blocks, both precisions
        dict(name="step_wavy4x128_f32", do="step", flow="wavy", n=128, M=0.5, Re=1e4, law="sutherland",
             limiter="minmod", precision="f32"),
        dict(name="step_wavy4x128_f64", do="step", flow="wavy", n=128, M=0.5, Re=1e4, law="sutherland",
             limiter="minmod", precision="f64"),
        # uneven blocks on a tree of interfaces with farfield faces: the largest
        # workload, and a smaller one in FP64
        dict(name="step_tree24_f32", do="step", flow="tree", layout=0, blocks=24, lo=16, hi=160, M=0.8, Re=5e4,
             law="sutherland", limiter="minmod", precision="f32"),
        dict(name="step_tree12_f64", do="step", flow="tree", layout=3, blocks=12, lo=16, hi=96, M=0.8, Re=5e4,
             law="sutherland", limiter="minmod", precision="f64"),
        # independent instances stepped together, each with its mu0 and dt
        dict(name="run_ensemble16x64_f32", do="run", flow="ensemble", blocks=16, n=64, layout=0, law="constant",
             limiter="minmod", precision="f32", steps=10, every=0),
        # the gradient of the kinetic energy after a number of steps
        dict(name="grad_tgv96_f32", do="grad", flow="tgv", n=96, M=0.3, Re=800.0, law="sutherland",
             limiter="minmod", precision="f32", steps=10, every=5),
        dict(name="grad_tgv48_f64", do="grad", flow="tgv", n=48, M=0.3, Re=800.0, law="sutherland",
             limiter="minmod", precision="f64", steps=20, every=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above (no name)."""
    do = rng.choice(["step", "step", "step", "run", "grad", "rhs"])
    c = dict(do=do, limiter=rng.choice(["minmod", "minmod", "vanleer"]), law=rng.choice(["sutherland", "constant"]),
             precision=rng.choice(["f32", "f64"]))
    if do == "step":
        flow = rng.choice(["tgv", "duct", "wavy", "tree"])
    elif do == "run":
        flow = rng.choice(["tgv", "ensemble", "wavy"])
    elif do == "grad":
        flow = rng.choice(["tgv", "wavy"])
    else:
        flow = "duct"
    c["flow"] = flow
    c["M"] = round(rng.uniform(0.1, 0.9), 3)
    c["Re"] = round(math.exp(rng.uniform(math.log(1e2), math.log(5e4))), 1)
    if flow == "tgv":
        c["n"] = _log_int(rng, 16, 96 if do != "step" else 160)
    elif flow == "wavy":
        c["n"] = _log_int(rng, 16, {"step": 128, "run": 64, "grad": 48}[do])
    elif flow == "duct":
        c["ni"], c["nj"], c["nk"] = (_log_int(rng, 8, 160) for _ in range(3))
    elif flow == "tree":
        c["blocks"] = rng.randint(2, 24)
        c["lo"], c["hi"] = 16, rng.randint(32, 128)
        c["layout"] = rng.randint(0, 9999)
    else:  # ensemble
        c["blocks"] = rng.randint(2, 32)
        c["n"] = _log_int(rng, 16, 64)
        c["layout"] = rng.randint(0, 9999)
        del c["M"], c["Re"]
    if do == "run":
        cells = sum(a * b * d for a, b, d in _shapes(c))
        c["steps"] = rng.randint(4, max(4, min(20, 45_000_000 // cells)))  # no more than the largest loop listed
        c["every"] = rng.choice([0, 1, 5])
    elif do == "grad":
        c["steps"] = rng.randint(2, 12)
        c["every"] = rng.randint(1, 6)
    return c


# ---------------------------------------------------------------------------
# inputs: per block q, kxyz, vol; links (target block, face, source block,
# face); boundary faces (block, face, kind).  Faces 0..5 = i min, i max, ...
# ---------------------------------------------------------------------------
def _tree_layout(case):
    """Block sizes and neighbours of the uneven tree: per-axis sizes uniform in
    [lo, hi], a random spanning tree of same-axis opposite-face interfaces."""
    rng = np.random.default_rng(case["layout"])
    lo, hi = case["lo"], case["hi"]
    sizes, nbrs = [list(rng.integers(lo, hi + 1, size=3))], [{}]
    for b in range(1, case["blocks"]):
        while True:
            parent, face = int(rng.integers(0, b)), int(rng.integers(0, 6))
            if face not in nbrs[parent]:
                break
        sz = list(sizes[parent])
        sz[face // 2] = int(rng.integers(lo, hi + 1))
        sizes.append(sz)
        nbrs.append({face ^ 1: (parent, face)})
        nbrs[parent][face] = (b, face ^ 1)
    return [tuple(int(s) + 2 * GHOST for s in sz) for sz in sizes], nbrs


def _shapes(case):
    """Padded extents of every block."""
    flow = case["flow"]
    if flow == "duct":
        return [tuple(case[a] + 2 * GHOST for a in ("ni", "nj", "nk"))]
    if flow == "tree":
        return _tree_layout(case)[0]
    nb = {"tgv": 1, "wavy": 4}.get(flow) or case["blocks"]
    return [(case["n"] + 2 * GHOST,) * 3] * nb


def _conserved(rho, u, v, w, p):
    return torch.stack([rho, rho * u, rho * v, rho * w, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v + w * w)])


def _taylor_green(n, M, noise, rnd):
    x = (torch.arange(n + 2 * GHOST, dtype=torch.float64, device="cuda") - GHOST + 0.5) * (2.0 * math.pi / n)
    X, Y, Z = torch.meshgrid(x, x, x, indexing="ij")
    p = 1.0 / GAMMA + (M * M / 16.0) * (torch.cos(2 * X) + torch.cos(2 * Y)) * (torch.cos(2 * Z) + 2.0)
    rho = p * GAMMA * (1 + noise * rnd(X.shape))
    p = p * (1 + noise * rnd(X.shape))
    u = M * torch.sin(X) * torch.cos(Y) * torch.cos(Z) + noise * M * rnd(X.shape)
    v = -M * torch.cos(X) * torch.sin(Y) * torch.cos(Z) + noise * M * rnd(X.shape)
    return _conserved(rho, u, v, noise * M * rnd(X.shape), p)


def _freestream(shape, M, noise, rnd):
    return _conserved(1 + noise * rnd(shape), M + noise * M * rnd(shape), noise * M * rnd(shape),
                      noise * M * rnd(shape), (1 + noise * rnd(shape)) / GAMMA)


def _uniform_metrics(shape, h):
    kxyz = torch.zeros((3, 3) + tuple(shape), dtype=torch.float64, device="cuda")
    for d in range(3):
        kxyz[d, d] = 1.0 / h
    return kxyz, torch.full(tuple(shape), h ** 3, dtype=torch.float64, device="cuda")


def _wavy_metrics(n, bi, bj, amp=0.05):
    """x = I h + s, y = J h + s, z = K h with s = amp sin(2 pi I/N) sin(2 pi J/N)."""
    N, e = 2 * n, GHOST
    h = om = 2.0 * math.pi / N
    ar = torch.arange(-e, n + e, dtype=torch.float64, device="cuda")
    I, J = (bi * n + ar)[:, None], (bj * n + ar)[None, :]
    a = amp * om * torch.cos(om * I) * torch.sin(om * J)  # ds/dI
    b = amp * om * torch.sin(om * I) * torch.cos(om * J)  # ds/dJ
    D = h * (h + a + b)
    kxyz = torch.zeros((3, 3, n + 2 * e, n + 2 * e, n + 2 * e), dtype=torch.float64, device="cuda")
    kxyz[0, 0] = ((h + b) / D)[:, :, None]
    kxyz[0, 1] = (-b / D)[:, :, None]
    kxyz[1, 0] = (-a / D)[:, :, None]
    kxyz[1, 1] = ((h + a) / D)[:, :, None]
    kxyz[2, 2] = 1.0 / h
    return kxyz, (D * h)[:, :, None].expand(n + 2 * e, n + 2 * e, n + 2 * e).contiguous()


def _time_step(q, kxyz, vol):
    """CFL / max over interior cells of sum_a (|u . k_a| + c |k_a|) / vol."""
    s = (slice(GHOST, -GHOST),) * 3
    rho = q[(0,) + s]
    vel = [q[(m + 1,) + s] / rho for m in range(3)]
    p = (GAMMA - 1.0) * (q[(4,) + s] - 0.5 * rho * sum(x * x for x in vel))
    c = torch.sqrt(GAMMA * p / rho)
    tot = 0.0
    for a in range(3):
        k = [kxyz[(a, m) + s] for m in range(3)]
        tot = tot + (sum(x * y for x, y in zip(vel, k))).abs() + c * torch.sqrt(sum(x * x for x in k))
    return CFL / float((tot / vol[s]).max())


class _Inputs:
    """qs, kxyz, vol per block; links; boundary faces; gas numbers; dt, mu0 per block."""


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 17)

    def rnd(shape):
        return torch.randn(tuple(shape), dtype=torch.float64, device="cuda", generator=gen)

    x = _Inputs()
    x.links, x.bcs = [], []
    x.limiter, x.law, x.precision = case["limiter"], case["law"], case["precision"]
    flow, shapes = case["flow"], _shapes(case)
    M, Re = case.get("M"), case.get("Re")
    x.mu0s = None
    if flow in ("tgv", "ensemble"):
        n = case["n"]
        Ms, Res = [M], [Re]
        if flow == "ensemble":
            lay = np.random.default_rng(case["layout"])
            Ms = [float(m) for m in lay.uniform(0.1, 0.9, case["blocks"])]
            Res = [float(r) for r in np.exp(lay.uniform(math.log(1e2), math.log(1e4), case["blocks"]))]
            x.mu0s = [m / r for m, r in zip(Ms, Res)]
        x.mu0 = Ms[0] / Res[0]
        x.qs = [_taylor_green(n, m, 0.005, rnd) for m in Ms]
        x.metrics = [_uniform_metrics(s, 2.0 * math.pi / n) for s in shapes]
        x.links = [(b, f, b, f ^ 1) for b in range(len(Ms)) for f in range(6)]
    else:
        x.mu0 = M / Re
        x.qs = [_freestream(s, M, 0.01, rnd) for s in shapes]
        if flow == "wavy":
            x.metrics = [_wavy_metrics(case["n"], b % 2, b // 2) for b in range(4)]
            for b in range(4):
                bi, bj = b % 2, b // 2
                i2, j2 = (1 - bi) + 2 * bj, bi + 2 * (1 - bj)
                x.links += [(b, f, s, f ^ 1) for f, s in enumerate((i2, i2, j2, j2, b, b))]
        elif flow == "duct":  # periodic along i, walls at the j faces, symmetry planes at the k faces
            x.metrics = [_uniform_metrics(shapes[0], 2.0 * math.pi / 128)]
            x.links = [(0, 0, 0, 1), (0, 1, 0, 0)]
            x.bcs = [(0, 2, WALL), (0, 3, WALL), (0, 4, SYMMETRY), (0, 5, SYMMETRY)]
        else:
            nbrs = _tree_layout(case)[1]
            x.metrics = [_uniform_metrics(s, 2.0 * math.pi / 128) for s in shapes]
            for b, nb in enumerate(nbrs):
                for f in range(6):
                    if f in nb:
                        x.links.append((b, f) + nb[f])
                    elif f ^ 1 not in nb:
                        x.links.append((b, f, b, f ^ 1))
                    else:
                        x.bcs.append((b, f, FARFIELD))
    x.q_inf = [1.0, M or 0.0, 0.0, 0.0, 1.0 / GAMMA / (GAMMA - 1.0) + 0.5 * (M or 0.0) ** 2]
    dts = [_time_step(q, k, v) for q, (k, v) in zip(x.qs, x.metrics)]
    x.dts = dts if flow == "ensemble" else None
    x.dt = dts[0] if flow == "ensemble" else min(dts)
    return x


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _config(x):
    from famrdp_jax_b200.core.constants import BCType, Face
    from famrdp_jax_b200.core.types import BlockTopology, Config, GasModel, SchemeChoice

    kinds = {FARFIELD: BCType.FARFIELD, WALL: BCType.WALL, SYMMETRY: BCType.SYMMETRY}
    topos = []
    for b in range(len(x.qs)):
        nb = {Face(f): (s, Face(sf), 0) for t, f, s, sf in x.links if t == b}
        bc = {f: BCType.CUT1TO1 for f in nb}
        for t, f, kind in x.bcs:
            if t == b:
                nb[Face(f)], bc[Face(f)] = None, kinds[kind]
        topos.append(BlockTopology(block_id=b, neighbors=nb, bc_type=bc))
    T0 = 1.0 / GAMMA
    gas = GasModel(gamma=GAMMA, R=1.0, mu0=x.mu0, T0=T0, Ts=T0 * 110.4 / 288.15, Pr_lam=PRANDTL, visc_law=x.law)
    return Config(gas=gas, scheme=SchemeChoice(reconstruct="muscl2", flux="roe", rk_order=3, limiter=x.limiter),
                  bc_params={f: {"q_inf": list(x.q_inf)} for f in Face} if x.bcs else {}, topology=tuple(topos),
                  ghost=GHOST, nan_check=True, cfl=CFL, precision=x.precision)


def prepare(case, seed):
    """State, configuration and plan: what a solver has in hand before its time loop."""
    from famrdp_jax_b200.core.types import Block, Metrics, State
    from famrdp_jax_b200.solver.step import StepPlan

    x = _inputs(case, seed)
    xyz = torch.zeros((3, 1, 1, 1), dtype=torch.float64, device="cuda")
    state = State(blocks=tuple(Block(q=q, xyz=xyz.expand((3,) + tuple(q.shape[1:]))) for q in x.qs),
                  metrics=tuple(Metrics(jac=v, kxyz=k, vol=v) for k, v in x.metrics))
    cfg = _config(x)
    plan = None
    if case["do"] != "rhs":
        plan = StepPlan(state, cfg)
        if x.mu0s is not None:
            plan.set_ensemble(x.mu0s, x.dts)
    return dict(case=case, state=state, cfg=cfg, plan=plan, dt=x.dt)


def run(s):
    case, state, cfg, dt = s["case"], s["state"], s["cfg"], s["dt"]
    if case["do"] == "step":
        from famrdp_jax_b200.solver.step import step

        return [b.q for b in step(state, cfg, dt, plan=s["plan"]).blocks]
    if case["do"] == "run":
        from famrdp_jax_b200.solver.run import run as time_loop

        final, log = time_loop(state, cfg, dt, case["steps"], plan=s["plan"], check_every=case["every"],
                               residual_every=case["every"])
        return [b.q for b in final.blocks] + [np.array([r for _, _, r in log.rows], dtype=np.float64)]
    if case["do"] == "grad":
        from famrdp_jax_b200.solver.adjoint import adjoint_kinetic_energy

        J, grads, dmu = adjoint_kinetic_energy(state, cfg, dt, case["steps"], case["every"], plan=s["plan"])
        return [J, list(grads), dmu]
    from famrdp_jax_b200.rhs.invscd import compute_invscd_rhs
    from famrdp_jax_b200.rhs.viscous import compute_viscous_rhs

    q, m = state.blocks[0].q, state.metrics[0]
    return [compute_invscd_rhs(q, m, ghost=GHOST, gamma=cfg.gas.gamma, reconstruct="muscl2", flux="roe",
                               limiter=cfg.scheme.limiter, precision=cfg.precision),
            compute_viscous_rhs(q, m, gas=cfg.gas, ghost=GHOST, precision=cfg.precision)]


def work(case):
    """Per padded cell: the state and the metrics (10 doubles) read and the
    result written once; about 1100 floating-point operations per right-hand
    side (three Roe faces at 250, the viscous fluxes and their divergence at
    300, the combine), and about three times that for its transpose."""
    cells = sum(a * b * c for a, b, c in _shapes(case))
    bytes_, flops = 160.0 * cells, 3 * 1100.0 * cells
    if case["do"] == "run":
        flops *= case["steps"]
    elif case["do"] == "grad":
        flops *= 4 * case["steps"]
    elif case["do"] == "rhs":
        bytes_, flops = 200.0 * cells, 1100.0 * cells
    return {"bytes": bytes_, "flops": flops}


# ---------------------------------------------------------------------------
# the same in plain torch, FP64
# ---------------------------------------------------------------------------
def _prims(q):
    r = q[0]
    u, v, w = q[1] / r, q[2] / r, q[3] / r
    return r, u, v, w, (GAMMA - 1.0) * (q[4] - 0.5 * r * (u * u + v * v + w * w))


def _limited(a, b, limiter):
    same = a * b > 0.0
    if limiter == "minmod":
        return torch.where(same, torch.where(a.abs() < b.abs(), a, b), torch.zeros_like(a))
    return torch.where(same, 2.0 * a * b / torch.where(same, a + b, torch.ones_like(a)), torch.zeros_like(a))


def _roe(L, R, n):
    def side(s):
        r, u, v, w, p = s
        E = p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v + w * w)
        un = u * n[0] + v * n[1] + w * n[2]
        F = [r * un, r * u * un + p * n[0], r * v * un + p * n[1], r * w * un + p * n[2], (E + p) * un]
        return [r, r * u, r * v, r * w, E], (E + p) / r, F

    UL, HL, FL = side(L)
    UR, HR, FR = side(R)
    sl, sr = torch.sqrt(L[0]), torch.sqrt(R[0])
    u, v, w, H = [(sl * a + sr * b) / (sl + sr) for a, b in zip(list(L[1:4]) + [HL], list(R[1:4]) + [HR])]
    q2 = u * u + v * v + w * w
    c2 = ((GAMMA - 1.0) * (H - 0.5 * q2)).clamp(min=1e-30)
    c = torch.sqrt(c2)
    un = u * n[0] + v * n[1] + w * n[2]
    eps = EPS_ENTROPY * (un.abs() + c)

    def fix(lam):
        return torch.where(lam.abs() >= eps, lam.abs(), 0.5 * (lam * lam / eps + eps))

    d = [b - a for a, b in zip(UL, UR)]
    dp = (GAMMA - 1.0) * (d[4] - u * d[1] - v * d[2] - w * d[3] + 0.5 * q2 * d[0])
    dun = d[1] * n[0] + d[2] * n[1] + d[3] * n[2] - un * d[0]
    rc = sl * sr * c * dun
    s1, s5 = fix(un - c) * (dp - rc) / (2.0 * c2), fix(un + c) * (dp + rc) / (2.0 * c2)
    a2, a23 = un.abs(), d[0] - dp / c2
    t = [d[m + 1] - h * d[0] - dun * n[m] for m, h in enumerate((u, v, w))]
    A = [s1 + s5 + a2 * a23]
    A += [s1 * (h - c * n[m]) + s5 * (h + c * n[m]) + a2 * (a23 * h + t[m]) for m, h in enumerate((u, v, w))]
    A.append(s1 * (H - c * un) + s5 * (H + c * un) + a2 * (a23 * 0.5 * q2 + u * t[0] + v * t[1] + w * t[2]))
    return torch.stack([0.5 * (a + b - e) for a, b, e in zip(FL, FR, A)])


def _invscd(q, kxyz, vol, limiter):
    pv = torch.stack(_prims(q))
    out = torch.zeros_like(q)
    for a in range(3):
        m = pv.shape[a + 1] - 3
        c0, c1, c2, c3 = (pv.narrow(a + 1, s, m) for s in range(4))
        L = c1 + 0.5 * _limited(c1 - c0, c2 - c1, limiter)
        R = c2 - 0.5 * _limited(c2 - c1, c3 - c2, limiter)
        nf = 0.5 * (kxyz[a].narrow(a + 1, 1, m) + kxyz[a].narrow(a + 1, 2, m))
        mag = torch.sqrt((nf * nf).sum(0))
        F = _roe(L.unbind(0), R.unbind(0), (nf / mag).unbind(0)) * mag
        div = F.narrow(a + 1, 1, m - 1) - F.narrow(a + 1, 0, m - 1)
        pad = [0, 0] * 3
        pad[2 * (2 - a)], pad[2 * (2 - a) + 1] = 2, 2
        out = out - torch.nn.functional.pad(div / vol.narrow(a, 2, m - 1), pad)
    return out


def _central(f, a):
    return 0.5 * (torch.roll(f, -1, a) - torch.roll(f, 1, a))


def _viscous(q, kxyz, mu0, law):
    r, u, v, w, p = _prims(q)
    T, T0 = p / r, 1.0 / GAMMA
    Ts = T0 * 110.4 / 288.15
    mu = mu0 * (torch.ones_like(T) if law == "constant" else (T / T0) ** 1.5 * (T0 + Ts) / (T + Ts))

    def grad(f):
        d = [_central(f, a) for a in range(3)]
        return [d[0] * kxyz[0, m] + d[1] * kxyz[1, m] + d[2] * kxyz[2, m] for m in range(3)]

    g, gT = [grad(f) for f in (u, v, w)], grad(T)
    div = g[0][0] + g[1][1] + g[2][2]
    tau = [[mu * (g[a][b] + g[b][a]) - (2.0 / 3.0 * mu * div if a == b else 0.0) for b in range(3)] for a in range(3)]
    kap = GAMMA / (GAMMA - 1.0) / PRANDTL * mu
    flux = tau + [[u * tau[0][m] + v * tau[1][m] + w * tau[2][m] + kap * gT[m] for m in range(3)]]
    rows = [sum(_central(f[m], a) * kxyz[a, m] for m in range(3) for a in range(3)) for f in flux]
    return torch.stack([torch.zeros_like(u)] + rows)


def _fill(qs, x):
    out = [q.clone() for q in qs]
    for t, f, s, sf in x.links:
        ax, n = f // 2, out[t].shape[f // 2 + 1]
        sax, sn = sf // 2, qs[s].shape[sf // 2 + 1]
        src = qs[s].narrow(sax + 1, GHOST if sf % 2 == 0 else sn - 2 * GHOST, GHOST)
        out[t].narrow(ax + 1, 0 if f % 2 == 0 else n - GHOST, GHOST).copy_(src)
    for b, f, kind in x.bcs:
        ax, n = f // 2, out[b].shape[f // 2 + 1]
        for o in range(GHOST):
            to, fr = (o, 2 * GHOST - 1 - o) if f % 2 == 0 else (n - 1 - o, n - 2 * GHOST + o)
            if kind == FARFIELD:
                val = torch.tensor(x.q_inf, dtype=torch.float64, device="cuda")[:, None, None]
            else:
                sign = [1.0, -1.0, -1.0, -1.0, 1.0] if kind == WALL else [1.0] * 5
                if kind == SYMMETRY:
                    sign[ax + 1] = -1.0
                val = out[b].select(ax + 1, fr) * torch.tensor(sign, dtype=torch.float64, device="cuda")[:, None, None]
            out[b].select(ax + 1, to).copy_(val)
    return out


def _step(qs, x, mu0s, dts):
    done = []
    for q, (kxyz, vol), mu0, dt in zip(_fill(qs, x), x.metrics, mu0s, dts):
        def L(y):
            return _invscd(y, kxyz, vol, x.limiter) + _viscous(y, kxyz, mu0, x.law)

        q1 = q + dt * L(q)
        q2 = 0.75 * q + 0.25 * (q1 + dt * L(q1))
        done.append(q / 3.0 + (2.0 / 3.0) * (q2 + dt * L(q2)))
    return done


def _interior(f):
    return f[..., GHOST:-GHOST, GHOST:-GHOST, GHOST:-GHOST]


def exact(case, seed):
    cells = sum(a * b * c for a, b, c in _shapes(case))
    if case["do"] == "grad" and cells > 1_200_000:
        return None
    x = _inputs(case, seed)
    nb = len(x.qs)
    mu0s, dts = x.mu0s or [x.mu0] * nb, x.dts or [x.dt] * nb
    if case["do"] == "rhs":
        (kxyz, vol), q = x.metrics[0], x.qs[0]
        return [_invscd(q, kxyz, vol, x.limiter), _viscous(q, kxyz, x.mu0, x.law)]
    if case["do"] == "step":
        return _step(x.qs, x, mu0s, dts)
    if case["do"] == "run":
        qs, rows = x.qs, []
        for n in range(1, case["steps"] + 1):
            new = _step(qs, x, mu0s, dts)
            if case["every"] and n % case["every"] == 0:
                d = [_interior(a - b).reshape(5, -1) / x.dt for a, b in zip(new, qs)]
                tot = sum(e.shape[1] for e in d)
                rows.append([math.sqrt(float(sum((e[m] * e[m]).sum() for e in d)) / tot) for m in range(5)])
            qs = new
        return qs + [np.array(rows, dtype=np.float64)]
    mu = torch.tensor(x.mu0, dtype=torch.float64, device="cuda", requires_grad=True)
    start = [q.clone().requires_grad_(True) for q in x.qs]
    qs = start
    for _ in range(case["steps"]):
        qs = torch.utils.checkpoint.checkpoint(lambda m, *y: tuple(_step(list(y), x, [m] * nb, dts)), mu, *qs,
                                               use_reentrant=False)
    J = sum((_interior(vol) * 0.5 * sum(_interior(q[m]) ** 2 for m in (1, 2, 3)) / _interior(q[0])).sum()
            for q, (_, vol) in zip(qs, x.metrics))
    grads = torch.autograd.grad(J, start + [mu])
    return [float(J), list(grads[:-1]), float(grads[-1])]
