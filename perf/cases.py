"""Performance cases of the swept1d framework: the calls its users make, over the sizes they make them at.

``listed()`` gives the fixed cases, ``draw(rng)`` further ones of the same ranges; ``prepare`` makes what
a program holds before the call, ``run`` makes one call through the package's public entry points,
``work`` counts what the call cannot do without and ``exact`` gives its result in plain 64-bit torch.

A case is a dict of plain values.  Its ``kind`` names the entry point:

* ``device``: ``Solver.run_device`` on a state resident on the GPU, restarted from the kept initial
  condition (a parameter study, or a step of a larger program);
* ``host``: ``Solver.run`` from a host initial condition to a host final state (a single run);
* ``batch``: ``Solver.run_batch_device`` on an ensemble of periodic KS domains of uneven length;
* ``closure_step``: ``Closure.step``, coarse KS steps corrected by the learned closure;
* ``closure_grad``: ``Closure.grad``, the loss and gradient of one training minibatch.
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

PROBLEMS = {"heat": 0, "ks": 1, "euler": 2}
ALGS = {"classic": 0, "swept": 1, "variant": 2}
BCS = {"default": 0, "mirror": 1, "periodic": 2}
COMPS = {"heat": 1, "ks": 1, "euler": 3}
# operations of one cell-update (a full time step of one cell); for Euler every term of a cell's two
# interfaces is shared with a neighbour, and a division or square root counts as one operation
FLOPS = {"heat": 4, "ks": 40, "euler": 212}
HEAT_ALPHA, HEAT_DX = 8.418e-5, 0.001
KS_DX, KS_DT = 0.5, 0.005
GAMMA, MGAMMA = 1.4, 0.4
CLOSURE_PARAMS = 5506
CLOSURE_FLOPS = 2 * (5 * 32 + 5 * 32 * 32 + 5 * 32) + 2 * 64 * 8  # per cell and step, three layers and two GELUs
KS_FLOPS_STEP = 40


def _sw():
    return importlib.import_module("1dsweptcuda_gb300")


def _gpu():
    return torch.device("cuda")


def _dtype(case):
    return torch.float64 if case["precision"] == 8 else torch.float32


# ------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # The smallest call: the size the reference's accuracy procedure runs (nx 1024, tpb 64), host to
        # host; a program that checks a time step or a boundary makes hundreds of them.
        dict(name="ks_f64_host_1k", kind="host", problem="ks", precision=8, alg="swept", bc="default", nx=1024,
             tpb=64, steps=500),
        # A small domain over many steps (the Heat benchmark configuration, 4096 periodic cells): latency
        # per level and per launch is all there is.
        dict(name="heat_f64_4k", kind="device", problem="heat", precision=8, alg="swept", bc="periodic", nx=4096,
             tpb=128, steps=4000, fo=0.1),
        # The headline configuration (2^20 cells, tpb 256, dx 0.5, dt 0.005) over a tenth of its horizon.
        dict(name="ks_f64_1m", kind="device", problem="ks", precision=8, alg="swept", bc="default", nx=1 << 20,
             tpb=256, steps=4000),
        # The large sizes of the reference's performance sweep, in both precisions.
        dict(name="ks_f32_4m", kind="device", problem="ks", precision=4, alg="swept", bc="default", nx=1 << 22,
             tpb=1024, steps=2048),
        dict(name="heat_f64_4m", kind="device", problem="heat", precision=8, alg="swept", bc="mirror", nx=1 << 22,
             tpb=512, steps=2000, fo=0.25),
        dict(name="heat_f32_4m", kind="device", problem="heat", precision=4, alg="swept", bc="mirror", nx=1 << 22,
             tpb=1024, steps=4096, fo=0.25),
        # Shock-tube runs: the large FP64 one, and an FP32 one of odd sizes (a tile width that is no power
        # of two, a step count that leaves classic steps over).
        dict(name="euler_f64_2m", kind="device", problem="euler", precision=8, alg="swept", bc="default", nx=1 << 21,
             tpb=512, steps=128),
        dict(name="euler_f32_odd", kind="device", problem="euler", precision=4, alg="swept", bc="default", nx=999936,
             tpb=384, steps=500),
        # The classic scheme, which every comparison runs beside the swept one: a launch per sub-step.
        dict(name="ks_f32_classic_1m", kind="device", problem="ks", precision=4, alg="classic", bc="default",
             nx=1 << 20, tpb=256, steps=1000),
        # The ensemble: domains of 2^10..2^16 cells (log-uniform), the tile width left to the autotuner.
        dict(name="ensemble_f32_1k", kind="batch", problem="ks", precision=4, alg="swept", domains=1024, lo=10, hi=16,
             steps=1000),
        # The closure: one segment of the certified coarse run (50 steps of 1024 domains), and one
        # minibatch of its training (64 of 512 samples, forward and backward).
        dict(name="closure_step_1k", kind="closure_step", domains=1024, n=1024, steps=50),
        dict(name="closure_grad_64", kind="closure_grad", samples=512, batch=64, n=1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choices(["device", "host", "batch", "closure_step", "closure_grad"], [12, 2, 2, 2, 1])[0]
    if kind in ("device", "host"):
        problem = rng.choice(["heat", "ks", "euler"])
        precision = rng.choice([4, 8])
        alg = rng.choices(["swept", "classic", "variant"], [6, 2, 1])[0]
        tpb = rng.choice([32, 64, 96, 128, 192, 256, 256, 384, 512, 640, 1024, 1024])
        top = 1 << (18 if kind == "host" else 21 if problem == "euler" else 22)
        tiles = max(2, _log_int(rng, 1024, top) // tpb)
        case = dict(kind=kind, problem=problem, precision=precision, alg=alg, bc="default", nx=tiles * tpb, tpb=tpb)
        if problem == "heat":
            case["bc"] = rng.choice(["mirror", "periodic"])
            case["fo"] = rng.choice([0.1, 0.25, 0.4])
        updates = {("heat", 8): 4e9, ("heat", 4): 8e9, ("ks", 8): 1e9, ("ks", 4): 3e9, ("euler", 8): 8e7,
                   ("euler", 4): 4e8}[problem, precision]
        if alg != "swept":
            updates /= 8
        limit = 1000 if alg == "classic" else 4000
        most = max(4, min(limit, int(updates / case["nx"])))
        case["steps"] = _log_int(rng, max(3, most // 16), most)
        return case
    if kind == "batch":
        lo = rng.choice([8, 9, 10])
        return dict(kind=kind, problem="ks", precision=rng.choice([4, 4, 8]), alg=rng.choice(["swept", "swept", "classic"]),
                    domains=_log_int(rng, 8, 512), lo=lo, hi=rng.choice([12, 14]), steps=_log_int(rng, 64, 500))
    if kind == "closure_step":
        return dict(kind=kind, domains=_log_int(rng, 8, 1024), n=128 * _log_int(rng, 1, 8), steps=_log_int(rng, 5, 50))
    batch = _log_int(rng, 16, 256)
    return dict(kind=kind, samples=512, batch=batch, n=128 * _log_int(rng, 2, 8))


# ----------------------------------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cpu")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _waves(n, g, wavelengths, amplitude):
    """Sum of cosines of the given wavelengths (cells; rounded to a whole number of periods over n), random phases."""
    x = torch.arange(n, device=_gpu(), dtype=torch.float64)
    out = torch.zeros_like(x)
    ph = torch.rand(len(wavelengths), generator=g, dtype=torch.float64) * 2 * math.pi
    am = 0.5 + torch.rand(len(wavelengths), generator=g, dtype=torch.float64)
    for w, p, a in zip(wavelengths, ph.tolist(), am.tolist()):
        periods = max(1, round(n / w))
        out += a * torch.cos((2 * math.pi * periods / n) * x + p)
    return out * (amplitude / math.sqrt(len(wavelengths)))


def _initial(case, seed):
    """The initial state in 64 bits on the GPU, (nx,) or for Euler (nx, 3), rounded to the case's precision."""
    g = _gen(seed)
    n, problem = case["nx"], case["problem"]
    if problem == "heat":  # temperatures in a bar: an offset and waves from a few cells to the whole bar
        u = 300.0 + _waves(n, g, [n, n / 3, n / 17, 1000, 200, 40, 11], 40.0)
    elif problem == "ks":  # flame-front ripples around the most unstable wavelength (18 cells at dx = 0.5)
        u = _waves(n, g, [n, n / 5, 150, 60, 31, 24, 18, 15], 1.4)
    else:
        # A shock tube in the middle of its run: constant states between jumps, half of the segments
        # crossed by smooth acoustic and entropy waves.
        k = 16
        rho = torch.empty(n, device=_gpu(), dtype=torch.float64)
        vel, prs = torch.empty_like(rho), torch.empty_like(rho)
        r = torch.rand(3, k, generator=g, dtype=torch.float64)
        ripple = _waves(n, g, [n / 4, n / 40, 64, 25], 0.03)
        cuts = [round(i * n / k) for i in range(k + 1)]
        for i in range(k):
            s = slice(cuts[i], cuts[i + 1])
            wave = ripple[s] if i % 2 else torch.zeros_like(ripple[s])
            rho[s] = (0.2 + 0.8 * float(r[0, i])) * (1.0 + wave)
            vel[s] = 0.3 * (float(r[1, i]) - 0.5) * (i % 4 != 0) + wave
            prs[s] = (0.2 + 0.8 * float(r[2, i])) * (1.0 + 1.4 * wave)
        u = torch.stack([rho, rho * vel, prs / MGAMMA + 0.5 * rho * vel * vel], dim=1)
    return u.to(_dtype(case)).to(torch.float64)


def _config(sw, case):
    kw = dict(alg=ALGS[case["alg"]], time_mode=sw.TIME_STEPS, n_steps=case["steps"])
    if case["kind"] == "batch":
        kw.update(tpb=0, dx=KS_DX, dt=KS_DT)
    else:
        kw.update(bc=BCS[case["bc"]], nx=case["nx"], tpb=case["tpb"])
        if case["problem"] == "heat":
            kw.update(dx=HEAT_DX, dt=case["fo"] * HEAT_DX * HEAT_DX / HEAT_ALPHA)
        elif case["problem"] == "ks":
            kw.update(dx=KS_DX, dt=KS_DT)
        else:
            kw.update(dt=0.1 / (case["nx"] - 2))  # dt/dx = 0.1 at the default dx = 1/(nx - 2)
    return sw.make_config(PROBLEMS[case["problem"]], case["precision"], **kw)


def _lengths(case):
    """The ensemble's domain lengths: part of its configuration, the same for every seed."""
    g = _gen(20261203 + case["domains"])
    e = torch.randint(case["lo"], case["hi"] + 1, (case["domains"],), generator=g)
    return (1 << e).numpy().astype(np.int64)


def _ensemble(case, seed):
    """Domain lengths and their states, grouped by length: [(domain indices, (count, n) state in 64 bits)]."""
    nx = _lengths(case)
    g = _gen(seed)
    groups = []
    for n in np.unique(nx):
        idx = np.nonzero(nx == n)[0]
        k = torch.arange(1, 9, dtype=torch.float64)
        a = torch.randn(len(idx), 8, generator=g, dtype=torch.float64) / k
        ph = torch.rand(len(idx), 8, generator=g, dtype=torch.float64) * 2 * math.pi
        th = 2 * math.pi * torch.outer(k, torch.arange(int(n), dtype=torch.float64) / float(n)).to(_gpu())
        ca, sa = (a * torch.cos(ph)).to(_gpu()), (a * torch.sin(ph)).to(_gpu())
        u = ca @ torch.cos(th) - sa @ torch.sin(th)
        groups.append((idx, u.to(_dtype(case)).to(torch.float64)))
    return nx, groups


def _concat(nx, groups, dtype):
    starts = np.concatenate([[0], np.cumsum(nx)[:-1]])
    out = torch.empty(int(nx.sum()), dtype=dtype, device=_gpu())
    for idx, u in groups:
        n = u.shape[1]
        at = torch.from_numpy(starts[idx]).to(_gpu())[:, None] + torch.arange(n, device=_gpu())[None, :]
        out[at.reshape(-1)] = u.to(dtype).reshape(-1)
    return out


def _theta(seed):
    """Closure parameters of the size training arrives at: He-scaled layers, an output layer near 0.1, scale 1e-3."""
    rng = np.random.default_rng(seed)
    w1 = rng.standard_normal(160) * math.sqrt(2.0 / 5)
    b1 = rng.standard_normal(32) * 0.1
    w2 = rng.standard_normal(5120) * math.sqrt(2.0 / 160)
    b2 = rng.standard_normal(32) * 0.1
    w3 = rng.standard_normal(160) * 0.1
    return np.concatenate([w1, b1, w2, b2, w3, [0.05], [1e-3]]).astype(np.float32)


def _coarse(domains, n, seed):
    """Coarse KS states (dx = 2): waves of 4 to 64 coarse cells, the scales of developed chaos."""
    g = _gen(seed)
    u = torch.zeros(domains, n, dtype=torch.float64)
    x = torch.arange(n, dtype=torch.float64)
    for w in (4.5, 6, 9, 16, 64):
        periods = max(1, round(n / w))
        ph = torch.rand(domains, 1, generator=g, dtype=torch.float64) * 2 * math.pi
        a = torch.randn(domains, 1, generator=g, dtype=torch.float64) * (0.25 if w < 5 else 0.8)
        u += a * torch.cos((2 * math.pi * periods / n) * x[None, :] + ph)
    return u.to(torch.float32)


def prepare(case, seed):
    sw = _sw()
    kind = case["kind"]
    state = {"case": case, "sw": sw, "solver": sw.Solver(0)}
    if kind == "device":
        u = _initial(case, seed).to(_dtype(case))
        if case["problem"] == "euler":  # device layout: (rho, rho u, E, pad)
            u = torch.cat([u, torch.zeros_like(u[:, :1])], dim=1).contiguous()
        state.update(cfg=_config(sw, case), ic=u, u=torch.empty_like(u))
    elif kind == "host":
        state.update(cfg=_config(sw, case), ic=_initial(case, seed).to(_dtype(case)).cpu().numpy().reshape(-1).copy())
    elif kind == "batch":
        nx, groups = _ensemble(case, seed)
        u = _concat(nx, groups, _dtype(case))
        cfg = _config(sw, case)
        if case["alg"] == "swept":  # the tuner's choice for this ensemble, as a program asks for it once
            t = state["solver"].tune(cfg, nx)
            cfg.tpb, cfg.threads = t.tile, t.threads
        state.update(cfg=cfg, nx=nx, ic=u, u=torch.empty_like(u))
    else:
        closure = importlib.import_module("1dsweptcuda_gb300.closure")
        state["net"] = closure.Closure(state["solver"], _theta(seed))
        if kind == "closure_step":
            u = _coarse(case["domains"], case["n"], seed).to(_gpu())
            state.update(ic=u, u=torch.empty_like(u))
        else:
            g = _gen(seed + 2)
            u = _coarse(case["samples"], case["n"], seed).to(_gpu())
            # the coarse step's defects: fields of the output scale's size, smooth like the input
            t = 1e-3 * (u * torch.roll(u, 1, 1) + 0.3 * torch.randn(u.shape, generator=g).to(_gpu()))
            rows = torch.randint(0, case["samples"], (case["batch"],), generator=g).numpy().astype(np.int64)
            state.update(u=u, target=t.contiguous(), rows=rows)
    torch.cuda.synchronize()
    return state


# -------------------------------------------------------------------------------------------------- run
def run(state):
    case, sw, solver = state["case"], state["sw"], state["solver"]
    kind = case["kind"]
    if kind == "host":
        return solver.run(state["cfg"], state["ic"])[0]
    if kind == "closure_grad":
        return state["net"].grad(state["u"], state["target"], state["rows"])
    u = state["u"]
    u.copy_(state["ic"])
    if kind == "device":
        solver.run_device(state["cfg"], u.data_ptr(), sw.native.torch_stream())
    elif kind == "batch":
        solver.run_batch_device(state["cfg"], state["nx"], u.data_ptr(), sw.native.torch_stream())
    else:
        state["net"].step(u, case["steps"], True)
    return u


# ------------------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind in ("device", "host"):
        cells = case["nx"]
        cell = case["precision"] * (4 if case["problem"] == "euler" and kind == "device" else COMPS[case["problem"]])
        return {"bytes": 2 * cells * cell, "flops": cells * case["steps"] * FLOPS[case["problem"]]}
    if kind == "batch":
        cells = int(_lengths(case).sum())
        return {"bytes": 2 * cells * case["precision"], "flops": cells * case["steps"] * FLOPS["ks"]}
    if kind == "closure_step":
        cells = case["domains"] * case["n"]
        return {"bytes": 8 * cells + 4 * CLOSURE_PARAMS,
                "flops": cells * case["steps"] * (CLOSURE_FLOPS + KS_FLOPS_STEP)}
    cells = case["batch"] * case["n"]
    return {"bytes": 8 * cells + 8 * CLOSURE_PARAMS, "flops": 3 * cells * CLOSURE_FLOPS}


# ------------------------------------------------------------------------------------------------ exact
def _heat64(case, u, prec):
    real = np.float64 if prec == 8 else np.float32
    dt = case["fo"] * HEAT_DX * HEAT_DX / HEAT_ALPHA
    ds = real(HEAT_DX)
    fou = float(real(HEAT_ALPHA)) * dt / float(ds * ds)
    fo, fo2 = float(real(fou)), float(real(1.0 - 2.0 * fou))
    periodic = case["bc"] == "periodic"
    for _ in range(case["steps"]):
        left, right = torch.roll(u, 1), torch.roll(u, -1)
        if not periodic:  # insulated ends: the neighbour inside, twice
            left[0], right[-1] = u[1], u[-2]
        u = fo * (left + right) + fo2 * u
    return u


def _ks_rhs64(u, c4, d2, d4):
    ll, l, r, rr = (torch.roll(u, s, -1) for s in (2, 1, -1, -2))
    return (r * r - l * l) * c4 + (l + r - 2 * u) * d2 + (ll - 4 * l + 6 * u - 4 * r + rr) * d4


def _ks64(u, steps, dx, dt, prec):
    real = np.float64 if prec == 8 else np.float32
    d = real(dx)
    c4, d2, d4 = (float(v) for v in (real(1) / (real(4) * d), real(1) / (d * d), real(1) / (d * d * d * d)))
    h, hh = float(real(dt)), float(real(dt * 0.5))
    for _ in range(steps):
        star = u - hh * _ks_rhs64(u, c4, d2, d4)
        u = u + (-h) * _ks_rhs64(star, c4, d2, d4)
    return u


def _euler_sum64(q, gam, mg):
    """Flux sums of cells 1 .. n-2 of q (3, n): (F_left + S_left) - F_right - S_right."""
    a, b = q[:, :-1], q[:, 1:]  # interface i between cells i and i + 1
    d = 2 * b[0] * a[0] * (b[2] - a[2]) + (a[1] * a[1] * b[0] - b[1] * b[1] * a[0])
    zero = torch.zeros_like(d[:1])
    da, db = torch.cat([zero, d[:-1]]), torch.cat([d[1:], zero])
    ra = torch.cat([q[0, :1], q[0, :-2]])  # density left of the interface's left cell
    rb = torch.cat([q[0, 2:], q[0, -1:]])

    def limited(cur, oth, num, den, dn):
        skip = (dn == 0) | (d == 0) | ((dn < 0) != (d < 0))
        f = 0.5 * torch.clamp(num / torch.where(skip, torch.ones_like(den), den), max=1.0)
        return torch.where(skip, cur, cur + f * (oth - cur))

    tl = limited(a, b, ra * d, b[0] * da, da)
    tr = limited(b, a, rb * d, a[0] * db, db)

    def pressure(s):
        return mg * (s[2] - 0.5 * s[1] * s[1] / s[0])

    ul, ur, pl, pr = tl[1] / tl[0], tr[1] / tr[0], pressure(tl), pressure(tr)
    f = torch.stack([tl[1] + tr[1], tl[1] * ul + tr[1] * ur + pl + pr,
                     tl[2] * ul + tr[2] * ur + ul * pl + ur * pr])
    rl, rr = torch.sqrt(tl[0]), torch.sqrt(tr[0])
    hd = 1.0 / (rl * rr * (rl + rr))
    hy, hz = (rl * tr[1] + rr * tl[1]) * hd, (rl * tr[2] + rr * tl[2]) * hd
    s = (torch.sqrt(mg * (hz - 0.5 * hy * hy) * gam) + hy.abs()) * (tl - tr)
    return f[:, :-1] + s[:, :-1] - f[:, 1:] - s[:, 1:]


def _euler64(case, u, prec):
    nx = case["nx"]
    real = np.float64 if prec == 8 else np.float32
    dx = float(real(1) / (real(nx) - real(2)))
    dtdx = float(real((0.1 / (nx - 2)) / dx))
    gam, mg = float(real(GAMMA)), float(real(MGAMMA))
    bd = torch.tensor([[1.0, 0.0, float(real(1) / real(MGAMMA))], [0.125, 0.0, float(real(0.1 / mg))]],
                      dtype=torch.float64, device=u.device)
    q = u.T.contiguous()
    q[:, 0], q[:, nx - 1] = bd[0], bd[1]
    for _ in range(case["steps"]):
        star = q.clone()
        star[:, 1:-1] += 0.25 * dtdx * _euler_sum64(q, gam, mg)
        q = q.clone()
        q[:, 1:-1] += 0.5 * dtdx * _euler_sum64(star, gam, mg)
    return q.T.contiguous()


def _net64(theta, u):
    """The closure network in 64 bits on its BF16-rounded weights: (output scale s) * net(u), and net(u)."""
    def rounded(x):
        return x + (x.detach().to(torch.float32).to(torch.bfloat16).to(torch.float64) - x.detach())

    w1 = rounded(theta[0:160]).reshape(32, 1, 5)
    w2 = rounded(theta[192:5312]).reshape(32, 32, 5)
    w3 = rounded(theta[5344:5504]).reshape(1, 32, 5)
    x = u[:, None, :]
    for w, b in ((w1, theta[160:192]), (w2, theta[5312:5344]), (w3, theta[5504:5505])):
        xp = torch.cat([x[:, :, -2:], x, x[:, :, :2]], dim=2)
        x = sum(torch.einsum("oi,bix->box", w[:, :, t], xp[:, :, t:t + x.shape[2]]) for t in range(5)) + b[None, :, None]
        if w is not w3:
            x = 0.5 * x * (1.0 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))
    return x[:, 0, :]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("device", "host"):
        u = _initial(case, seed)
        if case["problem"] == "heat":
            u = _heat64(case, u, case["precision"])
        elif case["problem"] == "ks":
            u = _ks64(u, case["steps"], KS_DX, KS_DT, case["precision"])
        else:
            u = _euler64(case, u, case["precision"])
            if kind == "device":
                u = torch.cat([u, torch.zeros_like(u[:, :1])], dim=1).contiguous()
        return u.reshape(-1).cpu().numpy() if kind == "host" else u
    if kind == "batch":
        nx, groups = _ensemble(case, seed)
        done = [(idx, _ks64(u, case["steps"], KS_DX, KS_DT, case["precision"])) for idx, u in groups]
        return _concat(nx, done, torch.float64)
    theta = torch.from_numpy(_theta(seed)).to(torch.float64).to(_gpu())
    if kind == "closure_step":
        scale = float(theta[5505])
        out = []
        for u in _coarse(case["domains"], case["n"], seed).to(torch.float64).to(_gpu()).split(128):
            for _ in range(case["steps"]):
                u = _ks64(u, 1, 2.0, 0.02, 4) + scale * _net64(theta, u)
            out.append(u)
        return torch.cat(out)
    state = prepare(case, seed)
    rows = torch.from_numpy(state["rows"]).to(_gpu())
    theta.requires_grad_(True)
    net = _net64(theta, state["u"][rows].to(torch.float64))
    loss = ((net - state["target"][rows].to(torch.float64) / theta[5505].detach()) ** 2).mean()
    loss.backward()
    grad = theta.grad.clone()
    grad[5505] = 0.0
    return grad, float(loss.detach())
