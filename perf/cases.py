"""What a user of this framework has it do, as measurable cases.

Every case goes through the package's public entry points: ``Solver`` (device-resident runs, the reference's
host-array calls), ``Batch``, ``FrozenMoodSteps`` (forward and backward) and the gate's training calls.  Sizes and
options are those of the repository's configurations, tests and benchmark, with odd sizes beside them.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same ranges, ``prepare`` makes what a user's
program holds before the call, ``run`` is one pass, ``work`` the bytes and flops of the algorithm, ``exact`` the
outputs in plain torch float64, written here from the method's definition.

Initial states are analytic problems whose parameters come from the seed, carried on for ``pre`` steps by a
first-order finite-volume scheme in torch, so that shocks, contacts and smooth parts are all there, as in a run
that has been going for a while; ``pre`` 0 is the start of a run.
"""
from __future__ import annotations

import importlib
import importlib.util
import json
import math
import sys
from decimal import Decimal, getcontext
from functools import lru_cache
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
DEV = "cuda"
F64 = torch.float64


def _package():
    """The package directory gp-mood_gb300/ as module gpmood_gb300."""
    if "gpmood_gb300" not in sys.modules:
        d = ROOT / "gp-mood_gb300"
        spec = importlib.util.spec_from_file_location("gpmood_gb300", d / "__init__.py",
                                                      submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["gpmood_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["gpmood_gb300"]


NEUMANN, PERIODIC, REFLECTIVE, DMR = 17, 18, 20, 35
GP_MOOD, NN_GP_MOOD = 2, 203
SSP_RK3, SSP_RK4 = 10, 12
EXACT, FAST = 0, 1
GAMMA = 1.4

# Problem -> domain and boundary condition (the configurations' own).
PROBLEMS = {"rp2d": ((1.0, 1.0), NEUMANN), "sedov": ((1.0, 1.0), REFLECTIVE), "dmr": ((4.0, 1.0), DMR),
            "vortex": ((10.0, 10.0), PERIODIC)}


def _solver_case(name, kind, problem, lf, nf, fp, steps, pre, mord=5, ngp=3, integrator=SSP_RK3, gated=False):
    return {"name": name, "kind": kind, "problem": problem, "lf": lf, "nf": nf, "fp": fp, "steps": steps, "pre": pre,
            "mord": mord, "ngp": ngp, "integrator": integrator, "gated": gated}


def listed():
    return [
        # The smallest call: a Fortran-style host loop of Setdt and time_stepping on its own arrays, in the default
        # (reference-rounding) mode, as the smoke test and a first port of a host code make it.
        _solver_case("host_48x40_exact", "host2", "rp2d", 48, 40, EXACT, 1, 60),
        # The four-quadrant Riemann problem at 256^2 on the device, in the middle of a run: ordinary size, latency and
        # MOOD passes share the time with the fluxes.
        _solver_case("rp2d_256_fast", "advance", "rp2d", 256, 256, FAST, 4, 150),
        # The benchmark's point blast at 2048^2, device-resident, from its start.
        _solver_case("sedov_2048_fast", "advance", "sedov", 2048, 2048, FAST, 2, 0),
        # A host program that owns its arrays (pinned): state in, state out each step, ragged grid.
        _solver_case("host_pinned_701x499_fast", "host1", "sedov", 701, 499, FAST, 1, 40),
        # Double Mach reflection at 512x128 as bench.py runs it, its first 30 steps: MOOD passes take the larger share.
        _solver_case("dmr_512x128_fast", "advance", "dmr", 512, 128, FAST, 30, 0),
        # The recorded reference runs' size, reference rounding, radius 2 with 3 Gauss points.
        _solver_case("rp2d_400_exact", "advance", "rp2d", 400, 400, EXACT, 1, 150),
        # Radius 1 with 2 Gauss points (the other half of the recorded runs), smooth periodic flow, ragged grid.
        _solver_case("vortex_r1_397x203_fast", "advance", "vortex", 397, 203, FAST, 4, 0, mord=3, ngp=2),
        # SSP-RK4 at 200^2, as the recorded radius-2 runs integrate.
        _solver_case("rp2d_rk4_200_fast", "advance", "rp2d", 200, 200, FAST, 2, 100, integrator=SSP_RK4),
        # An ensemble of problems of uneven size: load, advance, read back.
        {"name": "batch_48_fast", "kind": "batch", "count": 48, "smallest": 64, "largest": 256, "fp": FAST, "steps": 3},
        # Gradient of a functional through the steps (the adjoint's configuration): forward and backward.
        {"name": "adjoint_vortex_128", "kind": "adjoint", "problem": "vortex", "lf": 128, "nf": 128, "fp": EXACT,
         "steps": 5, "every": 5, "pre": 0},
        # The same double Mach reflection with the a-priori network gate in front of MOOD.
        _solver_case("dmr_gated_512x128_fast", "advance", "dmr", 512, 128, FAST, 30, 0, gated=True),
        # One mini-batch of the gate's training at its batch size: loss, gradient, Adam.
        {"name": "gate_train_4096", "kind": "train", "n": 4096},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "rp2d", "sedov", "host1", "dmr", "exact", "r1", "rk4", "batch", "adjoint", "gated",
                       "train"])
    if kind == "small":
        return _drop(_solver_case("", "host2", "rp2d", rng.randint(24, 96), rng.randint(24, 96), EXACT, 1, 60))
    if kind == "rp2d":
        n = _log_int(rng, 96, 640)
        return _drop(_solver_case("", "advance", "rp2d", n, n + rng.randint(-20, 20), FAST, rng.randint(2, 4), 150))
    if kind == "sedov":
        n = _log_int(rng, 300, 2000)
        return _drop(_solver_case("", "advance", "sedov", n, n + rng.randint(-30, 30), FAST, rng.randint(1, 2), 0))
    if kind == "host1":
        return _drop(_solver_case("", "host1", "sedov", _log_int(rng, 128, 900), _log_int(rng, 128, 900), FAST, 1, 40))
    if kind == "dmr" or kind == "gated":
        nf = rng.randint(64, 160)
        return _drop(_solver_case("", "advance", "dmr", 4 * nf + rng.randint(-3, 3), nf, FAST, rng.randint(10, 30), 0,
                                  gated=kind == "gated"))
    if kind == "exact":
        n = _log_int(rng, 64, 500)
        return _drop(_solver_case("", "advance", "rp2d", n, n + rng.randint(-9, 9), EXACT, 1, 150))
    if kind == "r1":
        return _drop(_solver_case("", "advance", "vortex", _log_int(rng, 64, 600), _log_int(rng, 64, 600), FAST,
                                  rng.randint(2, 4), 0, mord=3, ngp=2))
    if kind == "rk4":
        n = _log_int(rng, 100, 400)
        return _drop(_solver_case("", "advance", "rp2d", n, n + rng.randint(-9, 9), FAST, rng.randint(1, 2), 100,
                                  integrator=SSP_RK4))
    if kind == "batch":
        lo = rng.randint(32, 96)
        return {"kind": "batch", "count": rng.randint(8, 48), "smallest": lo, "largest": rng.randint(128, 256),
                "fp": FAST, "steps": rng.randint(1, 3)}
    if kind == "adjoint":
        steps = rng.randint(2, 6)
        return {"kind": "adjoint", "problem": "vortex", "lf": rng.randint(48, 160), "nf": rng.randint(48, 160),
                "fp": EXACT, "steps": steps, "every": rng.randint(1, steps), "pre": 0}
    return {"kind": "train", "n": _log_int(rng, 256, 65536)}


def _drop(case):
    return {k: v for k, v in case.items() if k != "name"}


# ---------------------------------------------------------------------------
# Inputs


def _gen(seed):
    return np.random.Generator(np.random.PCG64(int(seed)))


def _p2c(r, u, v, p):
    return torch.stack([r, r * u, r * v, p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)], dim=-1)


def _mesh(lf, nf, lx, ly):
    dx, dy = lx / lf, ly / nf
    x = torch.arange(-3, lf + 5, dtype=F64, device=DEV) * dx - dx / 2
    y = torch.arange(-3, nf + 5, dtype=F64, device=DEV) * dy - dy / 2
    return x[None, :].expand(nf + 8, lf + 8), y[:, None].expand(nf + 8, lf + 8), dx, dy


def _jitter(g, state, amount):
    """A primitive state with every nonzero entry moved by up to +-amount of itself."""
    return [v * (1.0 + amount * g.uniform(-1, 1)) for v in state]


def _quadrants(x, y, split, states):
    right, top = x > split[0], y > split[1]
    prim = []
    for k in range(4):
        bl, br, tl, tr = (torch.full_like(x, float(s[k])) for s in states)
        prim.append(torch.where(top, torch.where(right, tr, tl), torch.where(right, br, bl)))
    return _p2c(*prim)


def _initial(problem, lf, nf, seed, pre):
    """A padded state of the problem's kind, ghosts filled."""
    g = _gen(seed)
    (lx, ly), bc = PROBLEMS[problem]
    x, y, dx, dy = _mesh(lf, nf, lx, ly)
    if problem == "rp2d":  # 2DRP3 with its states and split moved a little
        states = [_jitter(g, s, 0.1) for s in ((0.138, 1.206, 1.206, 0.029), (0.5323, 0.0, 1.206, 0.3),
                                               (0.5323, 1.206, 0.0, 0.3), (1.5, 0.0, 0.0, 1.5))]
        U = _quadrants(x, y, (g.uniform(0.7, 0.85), g.uniform(0.7, 0.85)), states)
    elif problem == "sedov":  # E0, rho, p and the blast's place moved
        e0, r0, p0 = (1.0 * g.uniform(0.8, 1.2), g.uniform(0.8, 1.2), 1e-5 * g.uniform(0.8, 1.2))
        cx, cy = 0.5 + 0.1 * g.uniform(-1, 1), 0.5 + 0.1 * g.uniform(-1, 1)
        dr = 3.5 * min(dx, dy)
        inner = (x - cx) ** 2 + (y - cy) ** 2 < dr * dr
        p = torch.where(inner, torch.full_like(x, 0.4 * e0 / (math.pi * dr * dr)), torch.full_like(x, p0))
        U = _p2c(torch.full_like(x, r0), torch.zeros_like(x), torch.zeros_like(x), p)
    elif problem == "dmr":  # Mach-10 oblique shock, its foot moved by up to two cells
        post = y > (x - 1.0 / 6 - 2 * dx * g.uniform(-1, 1)) * math.sqrt(3.0)
        pre_s, post_s = (1.4, 0.0, 0.0, 1.0), (8.0, 7.1447096, -4.125, 116.5)
        U = _p2c(*(torch.where(post, torch.full_like(x, b), torch.full_like(x, a)) for a, b in zip(pre_s, post_s)))
    else:  # isentropic vortex: strength and place moved
        beta, cx, cy = g.uniform(4, 6), 5 + g.uniform(-1, 1), 5 + g.uniform(-1, 1)
        r2 = (x - cx) ** 2 + (y - cy) ** 2
        rho = (1 - 0.4 * beta * beta / (8 * 1.4 * math.pi ** 2) * torch.exp(1 - r2)) ** 2.5
        s = 0.5 * beta / math.pi * torch.exp(0.5 * (1 - r2))
        U = _p2c(rho, 1 - s * (y - cy), 1 + s * (x - cx), rho ** 1.4)
    U = _boundary(U.contiguous(), bc, dx, dy, 0.0)
    t = 0.0
    for _ in range(pre):
        U, dt = _first_order_step(U, bc, dx, dy, t)
        t += dt
    return U, float(t)


def _first_order_step(U, bc, dx, dy, t):
    """One explicit Euler step of first-order HLL finite volumes (how a state in mid-run is made)."""
    r = U[..., 0]
    u, v = U[..., 1] / r, U[..., 2] / r
    p = (GAMMA - 1) * (U[..., 3] - 0.5 * r * (u * u + v * v))
    c = torch.sqrt(GAMMA * p / r)
    dt = 0.4 / float(((u.abs() + c) / dx + (v.abs() + c) / dy).max())

    def flux(d, a, b):
        w = u if d == 0 else v
        push = torch.zeros_like(U)
        push[..., 1 + d] = p
        push[..., 3] = p * w
        F = U * w[..., None] + push
        sl = torch.minimum(w[a] - c[a], w[b] - c[b]).clamp(max=0.0)[..., None]
        sr = torch.maximum(w[a] + c[a], w[b] + c[b]).clamp(min=0.0)[..., None]
        return (sr * F[a] - sl * F[b] + sl * sr * (U[b] - U[a])) / (sr - sl)

    fx = flux(0, (slice(4, -4), slice(3, -4)), (slice(4, -4), slice(4, -3)))
    fy = flux(1, (slice(3, -4), slice(4, -4)), (slice(4, -3), slice(4, -4)))
    U = U.clone()
    U[4:-4, 4:-4] -= dt / dx * (fx[:, 1:] - fx[:, :-1]) + dt / dy * (fy[1:] - fy[:-1])
    return _boundary(U, bc, dx, dy, t + dt), dt


def _knobs(case):
    (lx, ly), bc = PROBLEMS[case["problem"]]
    k = dict(lf=case["lf"], nf=case["nf"], lx=lx, ly=ly, bc_type=bc, fp_mode=case["fp"], tmax=1.0e3)
    if "mord" in case:
        k.update(mord=case["mord"], ngp=case["ngp"], integrator=case["integrator"])
        if case["gated"]:
            k["method"] = NN_GP_MOOD
    return k


@lru_cache(maxsize=1)
def _gate_file():
    """The committed gate's parameters and logit threshold."""
    d = ROOT / "gp-mood_gb300" / "gates"
    p = np.loadtxt(d / "gate_sedov_rp2d3.txt", dtype=np.float32).ravel()
    return p, float(json.loads((d / "gate_sedov_rp2d3.json").read_text())["threshold"])


def _batch_inputs(case, seed):
    """Seeded four-quadrant Riemann problems of uneven size."""
    g = _gen(seed)
    sizes, states = [], []
    for i in range(case["count"]):
        # the ensemble's sizes are the case's own, its states the seed's
        lf, nf = (int(v) for v in _gen(1000 + i).integers(case["smallest"], case["largest"] + 1, size=2))
        quad = [(g.uniform(0.1, 2), g.uniform(-1.5, 1.5), g.uniform(-1.5, 1.5), g.uniform(0.02, 2)) for _ in range(4)]
        x, y, dx, dy = _mesh(lf, nf, 1.0, 1.0)
        U = _quadrants(x, y, (g.uniform(0.3, 0.8), g.uniform(0.3, 0.8)), quad)
        sizes.append((lf, nf))
        states.append(_boundary(U, NEUMANN, dx, dy, 0.0))
    return sizes, states


def _train_inputs(case, seed):
    """Normalised 9-point stencils, smooth or with a jump (the positive class), and weights in mid-training."""
    g = torch.Generator(device=DEV).manual_seed(int(seed))
    n = case["n"]

    def rnd(*s):
        return torch.rand(*s, generator=g, device=DEV, dtype=torch.float32)

    px = torch.tensor([0, -1, 1, 0, 0, -2, 2, 0, 0], dtype=torch.float32, device=DEV)
    py = torch.tensor([0, 0, 0, -1, 1, 0, 0, -2, 2], dtype=torch.float32, device=DEV)
    d = (rnd(n, 1) - 0.5) * px + (rnd(n, 1) - 0.5) * py
    y = (rnd(n) < 0.2).float()
    base = 0.1 + rnd(n, 4, 1)
    slope = 0.05 * (rnd(n, 4, 1) - 0.5)
    jump = (2 * rnd(n, 4, 1)) * (d > 0.3 * (rnd(n, 1) - 0.5)).float()[:, None] * y[:, None, None]
    q = base * (1 + slope * d[:, None]) + jump
    x = (q / q.abs().amax(dim=2, keepdim=True)).reshape(n, 36).contiguous()
    parts = []
    for fan_in, size in ((36, 64 * 36), (36, 64), (64, 64 * 64), (64, 64), (64, 64), (64, 1)):
        parts.append((2 * rnd(size) - 1) / math.sqrt(fan_in))
    p = torch.cat(parts)
    m = 1e-3 * (2 * rnd(p.numel()) - 1)
    v = 1e-6 * (0.5 + rnd(p.numel()))
    return p, m, v, x, y


def prepare(case, seed):
    P = _package()
    kind = case["kind"]
    if kind == "train":
        p, m, v, x, y = _train_inputs(case, seed)
        s = {"kind": kind, "n": case["n"], "p0": p, "m0": m, "v0": v, "x": x, "y": y,
             "p": torch.empty_like(p), "m": torch.empty_like(m), "v": torch.empty_like(v),
             "grad": torch.zeros_like(p), "loss": torch.zeros(1, device=DEV)}
        s["T"] = importlib.import_module("gpmood_gb300.nn_train")
        torch.cuda.synchronize()
        return s
    if kind == "batch":
        sizes, states = _batch_inputs(case, seed)
        host = [u.cpu().numpy() for u in states]
        return {"kind": kind, "batch": P.Batch(sizes, bc_type=NEUMANN, fp_mode=case["fp"], tmax=1.0e3), "host": host,
                "steps": case["steps"]}
    u, t = _initial(case["problem"], case["lf"], case["nf"], seed, case["pre"])
    s = {"kind": kind, "t": t, "steps": case["steps"]}
    solver = P.Solver(**_knobs(case))
    s["solver"] = solver
    if case.get("gated"):
        p, thr = _gate_file()
        solver.set_nn(p)
        solver.set_nn_threshold(thr)
    if kind == "host2":
        s["u"] = u.cpu().numpy()
        s["out"] = np.empty_like(s["u"])
    elif kind == "host1":
        s["u"] = u.cpu().pin_memory()
        s["out"] = torch.empty_like(s["u"]).pin_memory()
    elif kind == "adjoint":
        s["u"], s["every"] = u, case["every"]
        s["steps_fn"] = importlib.import_module("gpmood_gb300.adjoint").FrozenMoodSteps
    else:
        s["u"], s["out"] = u, torch.empty_like(u)
    torch.cuda.synchronize()
    return s


def run(s):
    kind = s["kind"]
    if kind == "advance":  # a device-resident run: load, advance, read back on the device
        s["solver"].set_state_dev(s["u"].data_ptr(), s["t"])
        s["solver"].advance(s["steps"])
        s["solver"].get_state_dev(s["out"].data_ptr())
        return {"u": s["out"]}
    if kind == "host2":  # the reference's two calls on a host program's arrays
        dt = s["solver"].Setdt(s["u"], 1.0)
        s["solver"].time_stepping(s["u"], s["out"], s["t"], dt)
        return {"u": s["out"], "dt": dt}
    if kind == "host1":  # both in one call, on pinned arrays
        dt = s["solver"].setdt_time_stepping_ptr(s["u"].data_ptr(), s["out"].data_ptr(), s["t"], 1.0)
        return {"u": s["out"], "dt": dt}
    if kind == "batch":
        b = s["batch"]
        for i, h in enumerate(s["host"]):
            b.set_state(i, h, 0.0)
        b.advance(s["steps"])
        return [b.get_state(i)[0] for i in range(len(s["host"]))]
    if kind == "adjoint":
        u0 = s["u"].detach().clone().requires_grad_(True)
        uN = s["steps_fn"].apply(u0, s["solver"], s["steps"], s["every"], s["t"])
        J = (uN[4:-4, 4:-4, 0] ** 2).sum()
        J.backward()
        return {"u": uN.detach(), "J": J.detach(), "grad": u0.grad}
    T = s["T"]
    for k in ("p", "m", "v"):
        s[k].copy_(s[k + "0"])
    stream = torch.cuda.current_stream().cuda_stream
    T.loss_grad(s["p"].data_ptr(), s["x"].data_ptr(), s["y"].data_ptr(), s["n"], s["grad"].data_ptr(),
                s["loss"].data_ptr(), 1.0, stream=stream)
    T.adam(s["p"].data_ptr(), s["grad"].data_ptr(), s["m"].data_ptr(), s["v"].data_ptr(), 100, 3e-3, stream=stream)
    return {k: s[k] for k in ("loss", "grad", "p", "m", "v")}


def work(case):
    """Algorithmic bytes and flops: every RK stage reconstructs 2 faces a cell (two states of 4 variables at ngp
    points from np cells), solves ngp Riemann problems a face (~100 flops) and updates the cell; the state is read and
    written once a step."""
    kind = case["kind"]
    if kind == "train":
        macs = 36 * 64 + 64 * 64 + 64
        return {"bytes": case["n"] * 37 * 4 + 7 * 6593 * 4, "flops": 3 * 2 * macs * case["n"]}
    if kind == "batch":
        sizes = [tuple(int(v) for v in _gen(1000 + i).integers(case["smallest"], case["largest"] + 1, size=2))
                 for i in range(case["count"])]
        cells, np_, ngp, stages = sum(a * b for a, b in sizes), 13, 3, 3
        steps = case["steps"]
    else:
        cells, steps = case["lf"] * case["nf"], case["steps"]
        np_, ngp = (13, 3) if case.get("mord", 5) == 5 else (5, case["ngp"])
        stages = 5 if case.get("integrator") == SSP_RK4 else 3
    face = 2 * 4 * ngp * (2 * np_ - 1) + ngp * 100 + 8 * ngp
    flops = cells * steps * stages * (2 * face + 60)
    if kind == "adjoint":
        flops *= 4  # the forward, its replay, and a backward of about twice the forward
    return {"bytes": cells * 32 * 2 * (2 if kind == "adjoint" else 1), "flops": flops}


# ---------------------------------------------------------------------------
# The method in plain torch float64 (GP weights in 50-digit decimals), for exact()

_ST = [(0, 0), (-1, 0), (0, 1), (1, 0), (0, -1), (-1, -1), (-1, 1), (1, 1), (1, -1), (0, -2), (-2, 0), (0, 2), (2, 0)]
_NP = {1: 1, 3: 5, 5: 13}


def _boundary(U, bc, dx, dy, t):
    """Ghost columns of interior rows, then ghost rows of every column; returns U, changed in place."""
    lf, nf = U.shape[1] - 8, U.shape[0] - 8
    rows = slice(4, 4 + nf)
    if bc == NEUMANN:
        U[rows, :4] = U[rows, 4:5]
        U[rows, lf + 4:] = U[rows, lf + 3:lf + 4]
        U[:4] = U[4:5]
        U[nf + 4:] = U[nf + 3:nf + 4]
    elif bc == PERIODIC:
        U[rows, :4] = U[rows, lf:lf + 4].clone()
        U[rows, lf + 4:] = U[rows, 4:8].clone()
        U[:4] = U[nf:nf + 4].clone()
        U[nf + 4:] = U[4:8].clone()
    elif bc == REFLECTIVE:
        fx = torch.tensor([1, -1, 1, 1], dtype=U.dtype, device=U.device)
        fy = torch.tensor([1, 1, -1, 1], dtype=U.dtype, device=U.device)
        U[rows, :4] = U[rows, 4:8].flip(1) * fx
        U[rows, lf + 4:] = U[rows, lf:lf + 4].flip(1) * fx
        U[:4] = U[4:8].flip(0) * fy
        U[nf + 4:] = U[nf:nf + 4].flip(0) * fy
    else:  # double Mach reflection
        post = _p2c(*(torch.tensor(v, dtype=F64, device=U.device) for v in (8.0, 7.1447096, -4.125, 116.5)))
        pre = _p2c(*(torch.tensor(v, dtype=F64, device=U.device) for v in (1.4, 0.0, 0.0, 1.0)))
        x = torch.arange(-3, lf + 5, dtype=F64, device=U.device) * dx - dx / 2
        y = torch.arange(-3, nf + 5, dtype=F64, device=U.device) * dy - dy / 2
        for cols in (slice(0, 4), slice(lf + 4, lf + 8)):
            behind = y[rows, None] > (x[None, cols] - 1.0 / 6) * math.sqrt(3.0)
            U[rows, cols] = torch.where(behind[..., None], post, pre)
        fy = torch.tensor([1, 1, -1, 1], dtype=U.dtype, device=U.device)
        U[:4] = torch.where((x > 1.0 / 6)[None, :, None], U[4:8].flip(0) * fy, post)
        xmin = 1.0 / 6 + 10.0 * t / (0.5 * math.sqrt(3.0)) + 1.0 / math.sqrt(3.0)
        U[nf + 4:] = torch.where((x < xmin)[None, :, None], post, pre)
    return U


def _erf(x):
    """erf by its Taylor series (|x| < 1 here)."""
    term = total = x
    n = 0
    while abs(term) > Decimal(10) ** -48:
        n += 1
        term = -term * x * x / n
        total += term / (2 * n + 1)
    return total * 2 / _PI.sqrt()


getcontext().prec = 60
_PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494459")


@lru_cache(maxsize=64)
def _gp_weights(lf, nf, lx, ly, ngp, ell_o_dx=12):
    """GP-SE prediction weights from cell averages to face Gauss points, and the second-derivative weights.
    Returns {order: [face L, T, R, B][gauss point][stencil point]}, Gauss weights, (d2x, d2y)."""
    D, s2 = Decimal, Decimal(2).sqrt()
    hx, hy = D(lx) / lf, D(ly) / nf
    ell = D(ell_o_dx) * min(hx, hy)

    def cov1(d, s):
        def part(a):
            return a * _erf(a) + (-a * a).exp() / _PI.sqrt()
        q = s2 * s
        return _PI.sqrt() * s * s * (part((d + 1) / q) + part((d - 1) / q) - 2 * part(d / q))

    def pre1(d, h):
        s = ell / h
        return (_PI / 2).sqrt() * s * (_erf((d + D("0.5")) / (s2 * s)) - _erf((d - D("0.5")) / (s2 * s)))

    def pre2(d, h):
        m, p, s = d - D("0.5"), d + D("0.5"), ell / h
        return (m * (-(m * m) / (2 * s * s)).exp() - p * (-(p * p) / (2 * s * s)).exp()) / (ell * ell)

    if ngp == 2:
        pts, gw = [-D("0.5") / D(3).sqrt(), D("0.5") / D(3).sqrt()], [0.5, 0.5]
    else:
        e = D("0.5") * (D(3) / 5).sqrt()
        pts, gw = [-e, D(0), e], [0.5 * 5 / 9, 0.5 * 8 / 9, 0.5 * 5 / 9]
    covx = {d: cov1(D(d), ell / hx) for d in range(-4, 5)}
    covy = {d: cov1(D(d), ell / hy) for d in range(-4, 5)}
    z, d2 = {1: [[[1.0] + [0.0] * 12] * ngp] * 4}, None
    for order in (3, 5):
        n = _NP[order]
        A = [[covx[_ST[a][0] - _ST[b][0]] * covy[_ST[a][1] - _ST[b][1]] for b in range(n)] for a in range(n)]
        rhs = []
        for face in range(4):
            for g in range(ngp):
                px, py = [(-D("0.5"), pts[g]), (pts[g], D("0.5")), (D("0.5"), pts[g]), (pts[g], -D("0.5"))][face]
                rhs.append([pre1(_ST[a][0] - px, hx) * pre1(_ST[a][1] - py, hy) for a in range(n)])
        if order == 3:
            rhs.append([pre2(D(_ST[a][0]), hx) * pre1(D(_ST[a][1]), hy) for a in range(n)])
            rhs.append([pre2(D(_ST[a][1]), hy) * pre1(D(_ST[a][0]), hx) for a in range(n)])
        sol = _solve(A, rhs)
        rows = [[float(v) for v in r] + [0.0] * (13 - n) for r in sol]
        if order == 3:
            d2 = (rows[-2][:5], rows[-1][:5])
        z[order] = [[[v / sum(rows[f * ngp + g]) for v in rows[f * ngp + g]] for g in range(ngp)] for f in range(4)]
    return z, gw, d2


def _solve(A, rhs):
    """x of A x = b for every b (Gaussian elimination; A is positive definite)."""
    n = len(A)
    M = [list(A[i]) + [b[i] for b in rhs] for i in range(n)]
    for i in range(n):
        for j in range(i + 1, n):
            f = M[j][i] / M[i][i]
            M[j] = [a - f * b for a, b in zip(M[j], M[i])]
    for i in reversed(range(n)):
        M[i] = [v / M[i][i] for v in M[i]]
        for j in range(i):
            f = M[j][i]
            M[j] = [a - f * b for a, b in zip(M[j], M[i])]
    return [[M[i][n + k] for i in range(n)] for k in range(len(rhs))]


def _hllc(uL, uR, d):
    """HLLC flux in direction d of states [..., 4]."""
    def prim(u):
        w, t = u[..., 1 + d] / u[..., 0], u[..., 2 - d] / u[..., 0]
        p = (GAMMA - 1) * (u[..., 3] - 0.5 * (u[..., 1] ** 2 + u[..., 2] ** 2) / u[..., 0])
        ok = (u[..., 0] > 0) & (p > 0)
        c = torch.sqrt(torch.where(ok, GAMMA * p / u[..., 0], torch.ones_like(p)))
        return w, t, p, c, ok

    def flux(u, w, p):
        f = u * w[..., None]
        n = torch.zeros_like(f)
        n[..., 1 + d] = p
        n[..., 3] = p * w
        return f + n

    wL, tL, pL, cL, okL = prim(uL)
    wR, tR, pR, cR, okR = prim(uR)
    SL, SR = torch.minimum(wL - cL, wR - cR), torch.maximum(wL + cL, wR + cR)
    aL, aR = uL[..., 0] * (SL - wL), uR[..., 0] * (SR - wR)
    us = (uL[..., 0] * wL * (SL - wL) - uR[..., 0] * wR * (SR - wR) + pR - pL) / (aL - aR)

    def star(u, w, t, p, S, a):
        e = u[..., 3] / u[..., 0] + (us - w) * (us + p / a)
        v = [None, us, t] if d == 0 else [None, t, us]
        st = torch.stack([torch.ones_like(us), v[1], v[2], e], dim=-1) * (a / (S - us))[..., None]
        return flux(u, w, p) + S[..., None] * (st - u)

    F = torch.where((us >= 0)[..., None], star(uL, wL, tL, pL, SL, aL), star(uR, wR, tR, pR, SR, aR))
    F = torch.where((SR < 0)[..., None], flux(uR, wR, pR), F)
    F = torch.where((SL >= 0)[..., None], flux(uL, wL, pL), F)
    return torch.where((okL & okR)[..., None], F, torch.full_like(F, float("nan")))


class _Method:
    """GP-MOOD steps on a padded float64 state [ny, nx, 4], from the method's definition."""

    def __init__(self, lf, nf, lx, ly, bc, mord, ngp):
        self.lf, self.nf, self.nx, self.ny, self.bc, self.mord = lf, nf, lf + 8, nf + 8, bc, mord
        self.dx, self.dy = lx / lf, ly / nf
        z, gw, d2 = _gp_weights(lf, nf, lx, ly, ngp)
        self.z = {o: torch.tensor(w, dtype=F64, device=DEV) for o, w in z.items()}
        self.gw = torch.tensor(gw, dtype=F64, device=DEV)
        self.d2 = torch.tensor(d2, dtype=F64, device=DEV)
        i = torch.arange(self.ny * self.nx, device=DEV).reshape(self.ny, self.nx)
        self.inner = i[4:-4, 4:-4].reshape(-1)
        self.faces = (i[4:-4, 3:-4].reshape(-1), i[3:-4, 4:-4].reshape(-1))
        self.is_inner = torch.zeros(self.ny * self.nx, dtype=torch.bool, device=DEV)
        self.is_inner[self.inner] = True
        self.off = torch.tensor([x + y * self.nx for x, y in _ST], device=DEV)

    def face_flux(self, u, low, d, order):
        """Quadrature fluxes [F, 4] of the faces whose low cells are `low`, from flat states u."""
        step = 1 if d == 0 else self.nx
        o = torch.minimum(order[low], order[low + step])
        parts, places = [], []
        for k in (1, 3, 5):
            sel = torch.nonzero(o == k).reshape(-1)
            for at in torch.split(sel, 1 << 19):
                n = _NP[k]
                zl, zh = self.z[k][2 if d == 0 else 1][:, :n], self.z[k][0 if d == 0 else 3][:, :n]
                c = low[at]
                uL = torch.einsum("gm,fmk->fgk", zl, u[c[:, None] + self.off[:n]])
                uR = torch.einsum("gm,fmk->fgk", zh, u[c[:, None] + step + self.off[:n]])
                parts.append(torch.einsum("g,fgk->fk", self.gw, _hllc(uL, uR, d)))
                places.append(at)
        where = torch.cat(places)
        return torch.cat(parts)[torch.argsort(where)]

    def update(self, u, fx, fy, c, dt):
        qx, qy = dt / self.dx, dt / self.dy
        return u[c] + qy * fy[c - self.nx] + qx * fx[c - 1] - qx * fx[c] - qy * fy[c]

    def troubled(self, uo, u, c):
        """DETECTION of cells c with updated values uo, from the stage input u."""
        p = (GAMMA - 1) * (uo[:, 3] - 0.5 * (uo[:, 1] ** 2 + uo[:, 2] ** 2) / uo[:, 0])
        bad = ~((uo[:, 0] > 0) & (p > 0))
        nx = self.nx
        L, R, B, T, C = u[c - 1], u[c + 1], u[c - nx], u[c + nx], u[c]
        r5 = torch.stack([v[:, 0] for v in (C, L, B, T, R)])
        mn, mx = r5.amin(0), r5.amax(0)
        dmp = ((mx - mn) > self.dx ** 3) & ((uo[:, 0] > mx) | (uo[:, 0] < mn))

        def pr(v):
            return (GAMMA - 1) * (v[:, 3] - 0.5 * (v[:, 1] ** 2 + v[:, 2] ** 2) / v[:, 0])
        div = 0.5 * ((R[:, 1] - L[:, 1]) / self.dx + (T[:, 2] - B[:, 2]) / self.dy) / C[:, 0]
        div = div - 0.5 * (C[:, 1] * (R[:, 0] - L[:, 0]) / self.dx + C[:, 2] * (T[:, 0] - B[:, 0]) / self.dy) / C[:, 0] ** 2
        mach = torch.sqrt((C[:, 1] ** 2 + C[:, 2] ** 2) / C[:, 0] ** 2 / (1.4 * pr(C) / C[:, 0]))
        pL, pR, pB, pT = pr(L), pr(R), pr(B), pr(T)
        grad = 0.5 * ((pR - pL).abs() / torch.minimum(pL, pR) / self.dx + (pT - pB).abs() / torch.minimum(pB, pT) / self.dy)
        h = max(self.dx, self.dy)
        shock = (div < -h * h) & (mach > 0.2) & (grad > 5.0)
        smooth = torch.zeros_like(bad)
        cross = torch.stack([c - 1, c, c + 1, c - nx, c + nx], dim=1)
        rho = u[cross[:, :, None] + self.off[:5], 0]
        for w in self.d2:
            dd = rho @ w
            lo, hi = dd.amin(1), dd.amax(1)
            smooth |= (lo * hi > -h) & ((torch.maximum(lo.abs(), hi.abs()) < h) | ((lo / hi).abs() >= 0.5))
        return bad | (dmp & shock & ~smooth)

    def stage(self, U, dt, t, frozen=None):
        """One Forward_Euler: (input with ghosts, output with ghosts, orders)."""
        U = _boundary(U.clone(), self.bc, self.dx, self.dy, t)
        u = U.reshape(-1, 4)
        order = torch.full((len(u),), self.mord, device=DEV)
        fx, fy = torch.zeros_like(u), torch.zeros_like(u)
        for f, d in ((fx, 0), (fy, 1)):
            f[self.faces[d]] = self.face_flux(u, self.faces[d], d, order)
        out = torch.zeros_like(u)
        cells = self.inner
        while True:
            uo = self.update(u, fx, fy, cells, dt)
            out[cells] = uo
            bad = cells[self.troubled(uo, u, cells) & (order[cells] > 1)]
            if not len(bad):
                break
            order[bad] = torch.where(order[bad] > 3, 3, 1)
            for f, d, step in ((fx, 0, 1), (fy, 1, self.nx)):
                low = torch.unique(torch.cat([bad, bad - step]))
                f[low] = self.face_flux(u, low, d, order)
            cells = torch.unique(torch.cat([bad, bad - 1, bad + 1, bad - self.nx, bad + self.nx]))
            cells = cells[self.is_inner[cells]]
        return U, _boundary(out.reshape(U.shape), self.bc, self.dx, self.dy, t), order

    def dt(self, U, cfl=0.8):
        r = U[..., 0]
        p = (GAMMA - 1) * (U[..., 3] - 0.5 * (U[..., 1] ** 2 + U[..., 2] ** 2) / r)
        c = torch.sqrt(GAMMA * p / r)
        a, b = (U[..., 1] / r).abs() + c, (U[..., 2] / r).abs() + c
        return cfl * float((1 / (a / self.dx + b / self.dy)).min())

    def rk3(self, U, t, dt):
        U0, U1, o1 = self.stage(U, dt, t)
        _, U2, o2 = self.stage(U1, dt, t + dt)
        _, U3, o3 = self.stage(0.75 * U0 + 0.25 * U2, dt, t + dt / 2)
        return U0 / 3 + 2 * U3 / 3, (o1, o2, o3)

    def rk4(self, U, t, dt):
        def inc(V):
            a, b, _ = self.stage(V, dt, t)
            return a, b - a
        U, F = inc(U)
        U1 = U + 0.391752226571890 * F
        U1, F = inc(U1)
        U2 = 0.444370493651235 * U + 0.555629506348765 * U1 + 0.368410593050371 * F
        U2, F = inc(U2)
        U3 = 0.620101851488403 * U + 0.379898148511597 * U2 + 0.251891774271694 * F
        U3, F3 = inc(U3)
        U4 = 0.178079954393132 * U + 0.821920045606868 * U3 + 0.544974750228521 * F3
        U4, F4 = inc(U4)
        return (0.517231671970585 * U2 + 0.096059710526147 * U3 + 0.063692468666290 * F3 + 0.386708617503269 * U4 +
                0.226007483236906 * F4)

    def frozen_steps(self, u0, t, dts, orders):
        """The steps with every dt and order held, differentiable; no DETECTION."""
        num = torch.arange(self.ny * self.nx, dtype=F64, device=DEV).reshape(self.ny, self.nx, 1).repeat(1, 1, 4)
        src = _boundary(num, PERIODIC, self.dx, self.dy, 0.0)[..., 0].long().reshape(-1)  # the vortex's boundaries

        def stage(u, dt, order):
            u = u[src]
            fl = []
            for d in (0, 1):
                f = torch.zeros_like(u)
                fl.append(f.index_put((self.faces[d],), self.face_flux(u, self.faces[d], d, order)))
            new = self.update(u, fl[0], fl[1], self.inner, dt)
            return u, torch.zeros_like(u).index_put((self.inner,), new)[src]

        u = u0.reshape(-1, 4)
        for dt, (a, b, c) in zip(dts, orders):
            base, s1 = stage(u, dt, a)
            _, s2 = stage(s1, dt, b)
            _, s3 = stage(0.75 * base + 0.25 * s2, dt, c)
            u = base / 3 + 2 * s3 / 3
        return u.reshape(u0.shape)


def _run_method(M, U, t, steps, rk4=False, dt=None):
    dts, orders = [], []
    for _ in range(steps):
        h = M.dt(U) if dt is None else dt
        if rk4:
            U = M.rk4(U, t, h)
        else:
            U, o = M.rk3(U, t, h)
            orders.append(o)
        dts.append(h)
        t += h
    return U, dts, orders


def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "batch":
        sizes, states = _batch_inputs(case, seed)
        return [_run_method(_Method(lf, nf, 1.0, 1.0, NEUMANN, 5, 3), u, 0.0, case["steps"])[0]
                for (lf, nf), u in zip(sizes, states)]
    if case.get("gated"):
        return None  # which cells start lowered is the BF16 network's decision: no such value in 64 bits
    (lx, ly), bc = PROBLEMS[case["problem"]]
    M = _Method(case["lf"], case["nf"], lx, ly, bc, case.get("mord", 5), case.get("ngp", 3))
    U, t = _initial(case["problem"], case["lf"], case["nf"], seed, case["pre"])
    if kind == "adjoint":
        UN, dts, orders = _run_method(M, U, t, case["steps"])
        u0 = U.clone().requires_grad_(True)
        J = (M.frozen_steps(u0, t, dts, orders)[4:-4, 4:-4, 0] ** 2).sum()
        J.backward()
        return {"u": UN, "J": J.detach(), "grad": u0.grad}
    UN, dts, _ = _run_method(M, U, t, case["steps"], rk4=case["integrator"] == SSP_RK4)
    return {"u": UN} if kind == "advance" else {"u": UN, "dt": dts[0]}


def _exact_train(case, seed):
    """The mini-batch in 64 bits: mean cross-entropy with logits, its gradient, one Adam step."""
    p, m, v, x, y = (a.double() for a in _train_inputs(case, seed))
    p = p.requires_grad_(True)
    shapes = ((64, 36), (64,), (64, 64), (64,), (64,), (1,))
    W, at = [], 0
    for s in shapes:
        n = math.prod(s)
        W.append(p[at:at + n].reshape(s))
        at += n
    h = torch.relu(x @ W[0].T + W[1])
    h = torch.relu(h @ W[2].T + W[3])
    zl = h @ W[4] + W[5]
    loss = torch.nn.functional.binary_cross_entropy_with_logits(zl, y)
    loss.backward()
    g = p.grad
    m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
    new = p.detach() - 3e-3 * (m / (1 - 0.9 ** 100)) / (torch.sqrt(v / (1 - 0.999 ** 100)) + 1e-8)
    return {"loss": loss.detach().reshape(1), "grad": g, "p": new, "m": m, "v": v}
