"""The work that users of the solver have it do, as measurable cases.

Every case calls the framework's public entry points: the PyTorch operators
``torch.ops.dense2d.{rhs, stage, steps, batched_steps}``, the host driver ``Solver``, and the
differentiable form ``Adjoint`` / ``AdjointStep``. A case names a benchmark's boundary rules and
geometry (2 Sedov, 4 Richtmyer-Meshkov, 5 double Mach reflection, 9 shock/vortex, 11 periodic
vortex, 13 Rayleigh-Taylor between walls, 14 periodic Richtmyer-Meshkov, 1 the vortex between
outflow sides), a scheme (splitting 101 LLF, 102 GLF, 103 Steger-Warming with reconstruction 251
upwind5, 253 WENO-JS5, 255 WENO-Z5; 104 characteristic WENO-Z; 105 AdaWENO) and a grid.

States are made on the GPU from the seed alone: smooth flow with a vortex and long waves, captured
shocks and contacts (a front a cell or two wide) or the stratified Rayleigh-Taylor column, as the
benchmark's runs have them in mid-flight. ``exact`` is a plain PyTorch float64 restatement of the
same scheme, ghost layers included.
"""
from __future__ import annotations

import importlib
import math
import random

import torch

dense = importlib.import_module("2dense_gb300")
ops = importlib.import_module("2dense_gb300.torch_ops")
adjoint = importlib.import_module("2dense_gb300.adjoint")

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # one right-hand side on the smallest grid of the batched sweep: launches and latency
        dict(name="rhs-vortex-64", kind="rhs", bench=11, split=101, recon=253, ni=64, nj=64),
        # one Runge-Kutta stage on a small odd grid, as a program with its own time loop calls it
        dict(name="stage-rm-203x97", kind="stage", bench=4, split=102, recon=251, ni=203, nj=97, irk=2),
        # the isentropic vortex at its usual resolution
        dict(name="steps-vortex-200", kind="steps", bench=11, split=101, recon=253, ni=200, nj=200, n=10),
        # the same run between outflow sides through the host driver: arrays in, steps, arrays out
        dict(name="driver-vortex-200", kind="driver", bench=1, split=101, recon=253, ni=200, nj=200, n=5),
        # a right-hand side of the blast problem, odd grid, Steger-Warming splitting
        dict(name="rhs-sedov-481x479", kind="rhs", bench=2, split=103, recon=255, ni=481, nj=479),
        # the double Mach reflection: a preview grid and the production grid
        dict(name="steps-dmr-480x120", kind="steps", bench=5, split=105, recon=0, ni=480, nj=120, n=10),
        dict(name="steps-dmr-1920x480", kind="steps", bench=5, split=105, recon=0, ni=1920, nj=480, n=4),
        # Rayleigh-Taylor between walls with the characteristic scheme
        dict(name="steps-rt-256x1024", kind="steps", bench=13, split=104, recon=0, ni=256, nj=1024, n=3),
        # the vortex on the largest grid of the resolution study
        dict(name="steps-vortex-2048", kind="steps", bench=11, split=101, recon=253, ni=2048, nj=2048, n=2),
        # a parameter sweep: instances of uneven size advanced together
        dict(name="batch-48", kind="batch", split=101, recon=255, count=48, nmin=64, nmax=512, n=2, sizes=7),
        # the adjoint of the vortex run: forward with checkpoints, loss, gradient
        dict(name="adjoint-vortex-256", kind="adjoint", bench=11, split=101, recon=253, ni=256, nj=256, n=12, every=6),
        # the transposed Jacobian of one characteristic right-hand side
        dict(name="vjp-rt-128x512", kind="vjp", bench=13, split=104, recon=0, ni=128, nj=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rhs", "stage", "steps", "steps", "steps", "driver", "batch", "adjoint", "vjp"])
    if kind == "batch":
        lo = rng.choice([64, 96, 128])
        return dict(kind=kind, split=rng.choice([101, 102]), recon=rng.choice([253, 255]),
                    count=_log(rng, 6, 60), nmin=lo, nmax=lo + 32 * rng.randint(1, 8), n=rng.randint(1, 3),
                    sizes=rng.randrange(1 << 20))
    split, recon = rng.choice([(101, 251), (101, 253), (101, 255), (102, 253), (102, 255), (103, 253), (103, 255),
                               (104, 0), (104, 0), (105, 0), (105, 0)])
    bench = rng.choice([1, 2, 4, 5, 9, 11, 11, 13, 14])
    cells = {"rhs": (3e3, 3e6), "stage": (3e3, 3e6), "steps": (8e3, 2e6), "driver": (4e3, 4e5),
             "adjoint": (2e3, 7e4), "vjp": (2e3, 3e5)}[kind]
    n = _log(rng, *cells)
    ratio = {5: 4.0, 13: 0.25, 4: 4.0, 9: 2.0}.get(bench, 1.0) * math.exp(rng.uniform(-0.5, 0.5))
    ni = max(17, int(math.sqrt(n * ratio)))
    nj = max(17, n // ni)
    c = dict(kind=kind, bench=bench, split=split, recon=recon, ni=ni, nj=nj)
    if kind == "stage":
        c["irk"] = rng.randint(1, 3)
    if kind in ("steps", "driver"):
        c["n"] = max(1, min(10, int(2e6 / n))) if kind == "steps" else rng.randint(1, 6)
    if kind == "adjoint":
        c["n"], c["every"] = rng.randint(2, 9), rng.randint(2, 5)
    return c


# -- configurations and inputs -----------------------------------------------------------------
def _geometry(case):
    """(dx, dy, gamma) of a benchmark on the case's grid."""
    ni, nj, b = case["ni"], case["nj"], case["bench"]
    w, h = {1: (10.0, 10.0), 11: (10.0, 10.0), 2: (1.2, 1.2), 4: (4.0, 1.0), 5: (4.0, 1.0), 9: (2.0, 1.0),
            14: (1.0, 1.0), 13: (0.25, 1.0)}[b]
    if b == 13:  # vertex grid
        return w / (ni - 1.0), h / (nj - 1.0), 5.0 / 3.0
    return w / ni, h / nj, 1.4


def _config(case):
    return dense.setup_config(dense.config_default(
        ni=case["ni"], nj=case["nj"], benchmark=case["bench"], splitting=case["split"], recon=case["recon"],
        cfl=0.4 if case["kind"] == "adjoint" else 0.5))


def _waves(X, Y, r, amp, top=3):
    """A few long waves of the unit square, periodic in both directions."""
    out = torch.zeros_like(X)
    for _ in range(4):
        kx, ky = r.randint(0, top), r.randint(1, top)
        out += amp * r.uniform(0.3, 1.0) * torch.sin(2 * math.pi * (kx * X + ky * Y + r.random()))
    return out


def _state(case, seed):
    """Conserved variables of the interior, (4, nj, ni)."""
    r = random.Random(1000003 * int(seed) + 17)
    ni, nj, b = case["ni"], case["nj"], case["bench"]
    g = _geometry(case)[2]
    x = (torch.arange(ni, dtype=F64, device=DEV) + 0.5) / ni
    y = (torch.arange(nj, dtype=F64, device=DEV) + 0.5) / nj
    Y, X = torch.meshgrid(y, x, indexing="ij")
    if b in (1, 11):  # the vortex in its unit stream
        eps, xc, yc = r.uniform(2.0, 5.0), r.uniform(0.35, 0.65), r.uniform(0.35, 0.65)
        dx, dy = 10.0 * (X - xc), 10.0 * (Y - yc)
        e = torch.exp(0.5 * (1.0 - dx * dx - dy * dy))
        T = 1.0 - (g - 1.0) * eps ** 2 / (8.0 * g * math.pi ** 2) * e * e
        u, v = 1.0 - eps / (2 * math.pi) * e * dy, 1.0 + eps / (2 * math.pi) * e * dx
        rho = T ** (1.0 / (g - 1.0)) * (1.0 + _waves(X, Y, r, 0.01))
        p = T ** (g / (g - 1.0))
    elif b == 13:  # heavy below light, the interface displaced
        yi = 0.5 + 0.02 * torch.cos(8 * math.pi * 0.25 * X) * r.uniform(0.5, 1.5) + _waves(X, 0 * Y, r, 0.002)
        s = 0.5 * (1.0 + torch.tanh((Y - yi) * nj / 1.5))
        rho = (2.0 - s) * (1.0 + _waves(X, Y, r, 0.01))
        p = torch.where(Y < 0.5, 2.0 * Y + 1.0, Y + 1.5)
        u = _waves(X, Y, r, 0.02)
        v = -0.05 * torch.cos(2 * math.pi * X) * torch.sqrt(g * p / rho) * torch.exp(-((Y - 0.5) * 8) ** 2) \
            + _waves(X, Y, r, 0.01)
    else:
        # a captured shock front, a second, curved front behind it and a contact; widths of a cell
        # or two, the states of a Mach 10 reflection for the double Mach problem, milder otherwise
        strong = b == 5
        x0 = r.uniform(0.6, 0.75) if strong else r.uniform(0.3, 0.6)
        slope = 0.25 / 3.0 ** 0.5 if strong else r.uniform(-0.1, 0.1)
        step = lambda d, n: 0.5 * (1.0 - torch.tanh(d * n / r.uniform(0.8, 1.3)))  # 1 where d < 0
        w = (X - 1.0).abs() if b == 14 else None  # periodic: the front's far side closes on itself
        front = step(X - x0 - slope * Y, ni)
        if w is not None:
            front = front * (1.0 - step(X - 0.05, ni))
        cx, rad = x0 - 0.12, r.uniform(0.12, 0.2)
        bow = torch.sqrt((X - cx) ** 2 + (Y / 3.0 * r.uniform(0.7, 1.0)) ** 2) - rad
        bow = step(bow, ni) * front
        slip = step(Y - 0.25 - 0.12 * torch.sin(6 * math.pi * X + 6.3 * r.random()), nj) * bow
        if strong:
            pre, post = (1.4, 0.0, 0.0, 1.0), (8.0, 7.145, -4.125, 116.5)
        else:
            pre, post = (1.0, 0.0, 0.0, 1.0), (1.8621, 0.8216, 0.0, 2.4583)
        rho, u, v, p = (a + (q - a) * front for a, q in zip(pre, post))
        rho = rho * (1.0 + 0.9 * bow) * (1.0 - 0.35 * slip)
        p = p * (1.0 + 1.3 * bow)
        u = u * (1.0 - 0.25 * bow + 0.2 * slip)
        v = v * (1.0 - 0.8 * bow)
        rho = rho * (1.0 + _waves(X, Y, r, 0.01))
        p = p * (1.0 + _waves(X, Y, r, 0.01))
        u, v = u + _waves(X, Y, r, 0.02), v + _waves(X, Y, r, 0.02)
    return torch.stack([rho, rho * u, rho * v, p / (g - 1.0) + 0.5 * rho * (u * u + v * v)]).contiguous()


def _padded(U):
    out = torch.zeros(4, U.shape[1] + 8, U.shape[2] + 8, dtype=F64, device=DEV)
    out[:, 4:-4, 4:-4] = U
    return out


def _instances(case):
    """The instances of a batch: square periodic grids, vortices and Richtmyer-Meshkov in turn."""
    r = random.Random(case["sizes"])
    sizes = [r.randrange(case["nmin"], case["nmax"] + 1, 32) for _ in range(case["count"])]
    return [dict(kind="steps", bench=11 if k % 2 == 0 else 14, split=case["split"], recon=case["recon"], ni=s, nj=s,
                 n=case["n"]) for k, s in enumerate(sizes)]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        inst = _instances(case)
        return dict(case=case, cfgs=[ops.config_tensor(_config(c)) for c in inst],
                    states=[_padded(_state(c, 100 * seed + k)) for k, c in enumerate(inst)])
    cfg = _config(case)
    U = _state(case, seed)
    st = dict(case=case, cfg=cfg)
    if kind in ("rhs", "stage", "steps"):
        st.update(cfg=ops.config_tensor(cfg), cons=_padded(U))
        if kind == "stage":
            # stages 2 and 3 start from another state than the step did, with the step's dt
            st.update(cons0=_padded(_state(case, seed + 500)), dt=0.2 * min(_geometry(case)[:2]) / 4.0)
    elif kind == "driver":
        st.update(solver=dense.Solver(cfg), cons=_fortran(_padded(U)), x=None, y=None)
        st["x"], st["y"] = _coordinates(case)
    else:
        st.update(adj=adjoint.Adjoint(cfg, checkpoint_every=case.get("every", 4)))
        if kind == "adjoint":
            st.update(u0=U.requires_grad_(True), target=_state(case, seed + 500)[0])
        else:
            r = torch.Generator(device="cpu").manual_seed(int(seed) + 5)
            st.update(u0=U, v=torch.randn(U.shape, generator=r, dtype=F64).to(DEV))
    return st


def _fortran(t):
    """A (nv, nj, ni) tensor as the host array a(i, j, v) of the Fortran driver."""
    return t.permute(2, 1, 0).cpu().numpy().copy(order="F")


def _coordinates(case):
    import numpy as np
    dx, dy, _ = _geometry(case)
    x = (np.arange(case["ni"]) + 0.5) * dx
    y = (np.arange(case["nj"]) + 0.5) * dy
    return (np.asfortranarray(np.broadcast_to(x[:, None], (case["ni"], case["nj"]))),
            np.asfortranarray(np.broadcast_to(y[None, :], (case["ni"], case["nj"]))))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rhs":
        return torch.ops.dense2d.rhs(state["cons"], state["cfg"])
    if kind == "stage":
        return torch.ops.dense2d.stage(state["cons"], state["cons0"], state["cfg"], case["irk"], state["dt"], 0.0)
    if kind == "steps":
        return torch.ops.dense2d.steps(state["cons"], state["cfg"], case["n"], 0.0)
    if kind == "batch":
        return torch.ops.dense2d.batched_steps(state["states"], state["cfgs"], case["n"])
    if kind == "driver":
        s = state["solver"]
        s.current_time, s.current_step = 0.0, 0
        s.upload(state["cons"], None, state["x"], state["y"])
        s.steps(case["n"])
        return s.download(with_prim=False), s.current_time
    if kind == "vjp":
        return state["adj"].rhs_vjp(state["u0"], state["v"])
    uT = adjoint.AdjointStep.apply(state["u0"], state["adj"], case["n"])
    loss = 0.5 * ((uT[0] - state["target"]) ** 2).sum()
    (grad,) = torch.autograd.grad(loss, state["u0"])
    return uT.detach(), loss.detach(), grad


# -- compulsory work ---------------------------------------------------------------------------
def _flops(case):
    """Operations of one cell-update (three stages) as the scheme writes them, adds, multiplies,
    divides and square roots one each; AdaWENO with every interface on its smooth branch."""
    if case["split"] == 104:
        return 6995.0
    if case["split"] == 105:
        return 1058.0 + 12 * 80.0
    base = {251: 1100.0, 253: 3748.0, 255: 4089.0}[case["recon"]]
    return base + (600.0 if case["split"] == 103 else 0.0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [work(c) for c in _instances(case)]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    cells, padded = case["ni"] * case["nj"], (case["ni"] + 8) * (case["nj"] + 8)
    f = _flops(case) * cells
    if kind == "rhs":
        return {"bytes": 32.0 * (padded + cells), "flops": f / 3}
    if kind == "stage":
        return {"bytes": 32.0 * padded * (2 if case["irk"] == 1 else 3), "flops": f / 3}
    if kind in ("steps", "driver"):
        return {"bytes": 64.0 * padded, "flops": f * case["n"]}
    if kind == "vjp":  # the right-hand side's terms and their transposed products
        return {"bytes": 96.0 * cells, "flops": f / 3 * 3}
    return {"bytes": 104.0 * cells, "flops": f * case["n"] * 3}


# -- the scheme in plain PyTorch ---------------------------------------------------------------
_SS = float(torch.tensor(1.0e-6, dtype=torch.float32))


def _betas(f):
    f0, f1, f2, f3, f4 = f
    return (13.0 / 12.0 * (f0 - 2 * f1 + f2) ** 2 + 0.25 * (f0 - 4 * f1 + 3 * f2) ** 2,
            13.0 / 12.0 * (f1 - 2 * f2 + f3) ** 2 + 0.25 * (f1 - f3) ** 2,
            13.0 / 12.0 * (f2 - 2 * f3 + f4) ** 2 + 0.25 * (3 * f2 - 4 * f3 + f4) ** 2)


def _candidates(f):
    f0, f1, f2, f3, f4 = f
    return ((2 * f0 - 7 * f1 + 11 * f2) / 6, (-f1 + 5 * f2 + 2 * f3) / 6, (2 * f2 + 5 * f3 - f4) / 6)


def _alphas(f, z):
    b = _betas(f)
    if not z:
        return [c / (_SS + q) ** 2 for c, q in zip((0.1, 0.6, 0.3), b)]
    tau = (b[2] - b[0]).abs()
    return [c * (1.0 + (tau / (_SS + q)) ** 2) for c, q in zip((0.1, 0.6, 0.3), b)]


def _weno(f, recon):
    if recon == 251:
        return (2 * f[0] - 13 * f[1] + 47 * f[2] + 27 * f[3] - 3 * f[4]) / 60
    a = _alphas(f, recon == 255)
    return sum(w * q for w, q in zip(a, _candidates(f))) / (a[0] + a[1] + a[2])


def _prims(U, g):
    rho, u, v = U[0], U[1] / U[0], U[2] / U[0]
    p = (g - 1.0) * (U[3] - 0.5 * rho * (u * u + v * v))
    return torch.stack([rho, u, v, p, torch.sqrt(g * p / rho)])


def _fixed(g, rho, u, v, p):
    return ([rho, rho * u, rho * v, p / (g - 1.0) + 0.5 * rho * (u * u + v * v)],
            [rho, u, v, p, math.sqrt(g * p / rho)])


_SIDES = {1: "PPEE", 2: "RERE", 4: "RREE", 5: "BTFE", 9: "RREE", 11: "PPPP", 13: "FFRR", 14: "PPPP"}


def _pad(case, A, axis, k, t):
    """The interior A with the four ghost layers of both sides of `axis` (1 y, 2 x); k 0 for the
    conserved variables, 1 for the primitives, which have ghosts of their own."""
    dx, dy, g = _geometry(case)
    b, ni = case["bench"], case["ni"]
    n = A.shape[axis]
    take = lambda q: A.narrow(axis, q, 1)
    flip = torch.ones(A.shape[0], 1, 1, dtype=F64, device=A.device)
    flip[3 - axis] = -1.0
    const = lambda s: torch.tensor(s[k], dtype=F64, device=A.device).view(-1, 1, 1)
    like = lambda s: s.expand_as(take(0))
    post, pre = _fixed(g, 8.0, 8.25 * math.sqrt(3.0) * 0.5, -8.25 * 0.5, 116.5), _fixed(g, 1.4, 0.0, 0.0, 1.0)
    x = ((torch.arange(ni, dtype=F64, device=A.device) + 0.5) * dx).view(1, 1, -1)
    out = []
    for hi in (0, 1):
        rule = _SIDES[b][(2 if axis == 2 else 0) + hi]
        inner = (lambda d: take(n - d)) if hi else (lambda d: take(d - 1))
        if rule == "P":
            side = [take(q) if hi else take(n - 1 - q) for q in range(4)]
        elif rule == "R":
            side = [flip * inner(q + 1) for q in range(4)]
        elif rule == "E":
            near, far, side = inner(1), inner(2), []
            for _ in range(4):
                near, far = near * 4.0 / 3.0 - far / 3.0, near
                side.append(near)
        elif rule == "B":
            side = [torch.where(x >= 1.0 / 6.0, flip * inner(q + 1), like(const(post))) for q in range(4)]
        else:
            if rule == "T":
                s = torch.where(x < 1.0 / 6.0 + (1.0 + 20.0 * t) / math.sqrt(3.0), const(post), const(pre))
            elif b == 13:
                s = const(_fixed(g, *((1.0, 0.0, 0.0, 2.5) if hi else (2.0, 0.0, 0.0, 1.0))))
            else:
                s = const(post)
            side = [like(s)] * 4
        out.append(side)
    return torch.cat(out[0][::-1] + [A] + out[1], dim=axis)


def _splits(case, U, W, d, speed):
    rho, u, v, p, a = W
    g = _geometry(case)[2]
    un, ut = (u, v) if d == 0 else (v, u)
    if case["split"] != 103:
        lam = un.abs() + a if case["split"] == 101 else speed
        z = torch.zeros_like(p)
        P = torch.stack([z, p if d == 0 else z, p if d == 1 else z, un * p])
        return 0.5 * ((un + lam) * U + P), 0.5 * ((un - lam) * U + P)
    both, ls = [], (un, un - a, un + a)
    for sg in (1.0, -1.0):
        p1, p2, p3 = ((l + sg * torch.sqrt(l * l + 0.125 ** 2)) / 2 for l in ls)
        c, A = rho / (2 * g), 2 * (g - 1.0) * p1
        fn = (A * un + p2 * ls[1] + p3 * ls[2]) * c
        ft = (A + p2 + p3) * ut * c
        e = ((g - 1.0) * p1 * (u * u + v * v) + 0.5 * p2 * (ls[1] ** 2 + ut * ut) + 0.5 * p3 * (ls[2] ** 2 + ut * ut)
             + (3.0 - g) * (p2 + p3) * a * a / (2 * (g - 1.0))) * c
        both.append(torch.stack([(A + p2 + p3) * c, fn, ft, e] if d == 0 else [(A + p2 + p3) * c, ft, fn, e]))
    return both


def _project(case, W, axis, n, d):
    """Left eigenvectors (rows: fields) and right eigenvectors at the faces' Roe states."""
    g = _geometry(case)[2]
    (rl, ul, vl, pl, _), (rr, ur, vr, pr, _) = (W.narrow(axis, 3 + s, n + 1) for s in (0, 1))
    hl, hr = (g / (g - 1.0) * p / r + 0.5 * (u * u + v * v) for p, r, u, v in ((pl, rl, ul, vl), (pr, rr, ur, vr)))
    wl, wr = torch.sqrt(rl), torch.sqrt(rr)
    mean = lambda a, b: (wl * a + wr * b) / (wl + wr)
    u, v, h = mean(ul, ur), mean(vl, vr), mean(hl, hr)
    q = 0.5 * (u * u + v * v)
    a = torch.sqrt((g - 1.0) * (h - q))
    b, o, z = (g - 1.0) / (a * a), torch.ones_like(u), torch.zeros_like(u)
    un, ut = (u, v) if d == 0 else (v, u)
    ex, ey = (1.0, 0.0) if d == 0 else (0.0, 1.0)
    left = [[0.5 * (b * q + un / a), -0.5 * (b * u + ex / a), -0.5 * (b * v + ey / a), 0.5 * b],
            [1.0 - b * q, b * u, b * v, -b],
            [-ut, ey * o, ex * o, z],
            [0.5 * (b * q - un / a), -0.5 * (b * u - ex / a), -0.5 * (b * v - ey / a), 0.5 * b]]
    right = [[o, u - ex * a, v - ey * a, h - a * un], [o, u, v, q], [z, ey * o, ex * o, ut],
             [o, u + ex * a, v + ey * a, h + a * un]]
    return left, right


def _rhs(case, U, t):
    dx, dy, g = _geometry(case)
    W = _prims(U, g)
    out = 0.0
    for d, h in ((0, dx), (1, dy)):
        axis, n = 2 - d, U.shape[2 - d]
        Wg = _pad(case, W, axis, 1, t)
        both = _splits(case, _pad(case, U, axis, 0, t), Wg, d, (W[1 + d].abs() + W[4]).max())
        faces = 0.0
        if case["split"] >= 104:
            left, right = _project(case, Wg, axis, n, d)
        for F, ks in zip(both, ((1, 2, 3, 4, 5), (6, 5, 4, 3, 2))):
            f = [F.narrow(axis, k, n + 1) for k in ks]
            if case["split"] < 104:
                faces = faces + _weno(f, case["recon"])
                continue
            cv = [_weno([sum(l[c] * m[c] for c in range(4)) for m in f], 255) for l in left]
            hc = torch.stack([sum(right[k][c] * cv[k] for k in range(4)) for c in range(4)])
            if case["split"] == 105:
                a = _alphas([Wg[0].narrow(axis - 1, k, n + 1) + m[1 + d] for k, m in zip(ks, f)], True)
                s = a[0] + a[1] + a[2]
                smooth = sum(w * q for w, q in zip(a, _candidates(f))) / s
                hc = torch.where(1.0 / (1.0 + (s - 1.0) ** 2) > 0.5, smooth, hc)
            faces = faces + hc
        out = out - (faces.narrow(axis, 1, n) - faces.narrow(axis, 0, n)) / h
    return out


_COEF = {1: (0.0, 1.0, 1.0, 1.0), 2: (0.75, 0.25, 0.25, 0.25),
         3: (1.0 / 3.0, 2.0 / 3.0, 2.0 / 3.0, float(torch.tensor(2.0 / 3.0, dtype=torch.float32)))}


def _dt(case, U, cfl):
    dx, dy, g = _geometry(case)
    W = _prims(U, g)
    ex, ey = dx / (W[1].abs() + W[4]).max(), dy / (W[2].abs() + W[4]).max()
    return cfl * ex * ey / (ex + ey)


def _stage(case, U, U0, irk, dt, t):
    a, b, c, f = _COEF[irk]
    V = a * U0 + b * U + c * dt * _rhs(case, U, t)
    if case["bench"] == 13:  # gravity along y
        z = torch.zeros_like(U[0])
        V = V + f * dt * torch.stack([z, z, U[0], U[2]])
    return V


def _step(case, U, t, cfl):
    """(the new state, dt, the last stage's input)"""
    dt = _dt(case, U, cfl)
    V, last = U, U
    for irk in (1, 2, 3):
        last, V = V, _stage(case, V, U, irk, dt, t)
    return V, dt, last


def _with_ghosts(case, given, U, last, t):
    """The padded result: ghosts of the last stage's input, on periodic grids of the result
    itself; the corners as they were given."""
    out = given.clone()
    out[:, 4:-4, 4:-4] = U
    src = U if _SIDES[case["bench"]] == "PPPP" else last
    P = _pad(case, src, 2, 0, t)
    out[:, 4:-4, :4], out[:, 4:-4, -4:] = P[:, :, :4], P[:, :, -4:]
    P = _pad(case, src, 1, 0, t)
    out[:, :4, 4:-4], out[:, -4:, 4:-4] = P[:, :4], P[:, -4:]
    return out


def _advance(case, given, n):
    U, t, last, t_last = given[:, 4:-4, 4:-4], 0.0, None, 0.0
    for _ in range(n):
        t_last = t
        U, dt, last = _step(case, U, t, 0.5)
        t = t + float(dt)
    return _with_ghosts(case, given, U, last, t_last), t


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_advance(c, _padded(_state(c, 100 * seed + k)), case["n"])[0] for k, c in enumerate(_instances(case))]
    U = _state(case, seed)
    if kind == "rhs":
        return _rhs(case, U, 0.0)
    if kind == "stage":
        U0 = _state(case, seed + 500)
        dt = _dt(case, U, 0.5) if case["irk"] == 1 else torch.tensor(0.2 * min(_geometry(case)[:2]) / 4.0, dtype=F64, device=DEV)
        return _with_ghosts(case, _padded(U), _stage(case, U, U0, case["irk"], dt, 0.0), U, 0.0), dt
    if kind == "steps":
        return _advance(case, _padded(U), case["n"])[0]
    if kind == "driver":
        out, t = _advance(case, _padded(U), case["n"])
        return _fortran(out), t
    U = U.requires_grad_(True)
    if kind == "vjp":
        r = torch.Generator(device="cpu").manual_seed(int(seed) + 5)
        v = torch.randn(U.shape, generator=r, dtype=F64).to(DEV)
        s = (_rhs(case, U, 0.0) * v).sum()
        return torch.autograd.grad(s, U)[0], float(s)
    from torch.utils.checkpoint import checkpoint
    # start times enter as values: the double Mach problem's top state is piecewise constant in time
    V, t = U, 0.0
    for _ in range(case["n"]):
        start = t
        V, dt = checkpoint(lambda W: _step(case, W, start, 0.4)[:2], V, use_reentrant=False)
        t = t + float(dt)
    loss = 0.5 * ((V[0] - _state(case, seed + 500)[0]) ** 2).sum()
    return V.detach(), loss.detach(), torch.autograd.grad(loss, U)[0]
