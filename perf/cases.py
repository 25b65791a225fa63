"""The work a program has this framework do, as cases that can be timed and compared.

Each case is one pass through the public entry points: the program's state goes in from the host
buffers it holds, a run of time steps (or training iterations) is done, and the whole result comes
back.  ``exact`` restates every scheme in plain 64-bit torch, without the framework.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from hyperflow_gb300 import BatchSolver, CartSolver, UnsSolver, cases
from hyperflow_gb300.learned import LearnedSolver, init_params

GAMMA = 1.4


def listed():
    return [
        # an interactive loop on the reference's smallest shipped case size: the host reads dt each step
        {"name": "tube_100x5_steps", "kind": "step", "nx": 100, "ny": 5, "scheme": "MUSCLHancock",
         "limiter": "VanLeer", "steps": 32},
        # the reference's first configuration: 256^2, 200 steps, in the device loop
        {"name": "quad_256_godunov", "kind": "run", "nx": 256, "ny": 256, "scheme": "Godunov", "limiter": "",
         "steps": 200},
        # an ordinary single block of sizes that divide no tile
        {"name": "quad_1000x777_vanleer", "kind": "run", "nx": 1000, "ny": 777, "scheme": "MUSCLHancock",
         "limiter": "VanLeer", "steps": 20},
        # a large first-order run, ragged
        {"name": "quad_2047x1999_godunov", "kind": "run", "nx": 2047, "ny": 1999, "scheme": "Godunov",
         "limiter": "", "steps": 20},
        # the largest single block of the benchmark
        {"name": "quad_4096_minbee", "kind": "run", "nx": 4096, "ny": 4096, "scheme": "MUSCLHancock",
         "limiter": "MinBee", "steps": 10},
        # the headline: the Mach 3 forward-facing step at dx = 1/1365, on a developed flow
        {"name": "ffs_1365_minbee", "kind": "ffs", "h": 1365, "limiter": "MinBee", "steps": 16, "io": False},
        # a host program that keeps its state in pinned memory and steps through hf_step_io
        {"name": "ffs_455_step_io", "kind": "ffs", "h": 455, "limiter": "MinBee", "steps": 12, "io": True},
        # many small independent problems at once
        {"name": "batch_24_minbee", "kind": "batch", "count": 24, "lo": 64, "hi": 384, "scheme": "MUSCLHancock",
         "limiter": "MinBee", "steps": 100},
        # a triangle mesh with the reference's bit-exact per-pair fluxes (the default mode)
        {"name": "uns_120k_pairs", "kind": "uns", "cells": 120_000, "edge": False, "steps": 200},
        # the ~1M-triangle mesh, one flux per edge
        {"name": "uns_1m_edges", "kind": "uns", "cells": 1_000_000, "edge": True, "steps": 100},
        # the learned coarse solver, run to an end time
        {"name": "learned_512_run", "kind": "learned", "n": 512, "steps": 60},
        # its training iterations
        {"name": "learned_256_train", "kind": "train", "n": 256, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "run", "run", "run", "ffs", "batch", "uns", "uns", "learned", "train"])
    scheme, limiter = rng.choice([("Godunov", ""), ("MUSCLHancock", "MinBee"), ("MUSCLHancock", "VanLeer")])
    if kind == "step":
        return {"kind": kind, "nx": _log(rng, 8, 400), "ny": _log(rng, 4, 200), "scheme": scheme,
                "limiter": limiter, "steps": rng.randint(8, 40)}
    if kind == "run":
        nx, ny = _log(rng, 64, 3600), _log(rng, 64, 3600)
        return {"kind": kind, "nx": nx, "ny": ny, "scheme": scheme, "limiter": limiter,
                "steps": max(4, min(200, int(6e7 / (nx * ny))))}
    if kind == "ffs":
        h = 5 * _log(rng, 13, 260)
        return {"kind": kind, "h": h, "limiter": limiter or "MinBee", "io": rng.random() < 0.4,
                "steps": max(4, min(100, int(4e7 / (2.52 * h * h))))}
    if kind == "batch":
        hi = _log(rng, 80, 500)
        return {"kind": kind, "count": _log(rng, 2, 40), "lo": max(16, hi // 6), "hi": hi, "scheme": scheme,
                "limiter": limiter, "steps": rng.randint(40, 100)}
    if kind == "uns":
        cells = _log(rng, 2_000, 900_000)
        return {"kind": kind, "cells": cells, "edge": rng.random() < 0.5,
                "steps": max(20, min(200, int(6e7 / cells)))}
    if kind == "learned":
        return {"kind": kind, "n": _log(rng, 48, 640), "steps": rng.randint(12, 60)}
    return {"kind": kind, "n": _log(rng, 32, 300), "steps": rng.randint(2, 8)}


# --- inputs ------------------------------------------------------------------------------------

def _cons(r, u, v, p):
    return torch.stack([r, r * u, r * v, p / (GAMMA - 1.0) + 0.5 * r * (u * u + v * v)])


def _flow(x, y, rng):
    """Primitive fields at (x, y) in the unit square: a four-quadrant Riemann problem drawn as the
    batched workload's (split in [0.3, 0.7]^2, rho in [0.1, 2], p in [0.1, 10], u and v in [-1, 1])
    under smooth waves of a few per cent."""
    sx, sy = rng.uniform(0.3, 0.7, 2)
    q = [torch.from_numpy(rng.uniform(a, b, 4)).to(x) for a, b in ((0.1, 2), (-1, 1), (-1, 1), (0.1, 10))]
    at = (x >= sx).long() + 2 * (y >= sy).long()
    w = [k[at] for k in q]
    for n, k in ((0, 0), (1, 3)):
        ph = rng.uniform(0, 2 * math.pi, 4)
        f = rng.integers(1, 7, 4)
        wave = torch.sin(2 * math.pi * f[0] * x + ph[0]) * torch.sin(2 * math.pi * f[1] * y + ph[1])
        w[k] = w[k] * (1 + 0.04 * wave)
        w[n + 1] = w[n + 1] + 0.03 * torch.sin(2 * math.pi * (f[2] * x + f[3] * y) + ph[2])
    return w


def _grid(nx, ny):
    x = (torch.arange(nx, dtype=torch.float64, device="cuda") + 0.5) / nx
    y = (torch.arange(ny, dtype=torch.float64, device="cuda") + 0.5) / ny
    return x[None, :].expand(ny, nx), y[:, None].expand(ny, nx)


def _pad(U, g):
    return torch.nn.functional.pad(U[None], (g, g, g, g), mode="replicate")[0]


def _pinned(U):
    out = torch.empty(U.shape, dtype=U.dtype, pin_memory=True)
    out.copy_(U)
    return out.numpy()


@functools.lru_cache(maxsize=2)
def _developed(limiter):
    """The forward-facing step's flow at t = 1.14 on a coarse mesh (dx = 1/65): bow shock,
    reflections and subsonic pockets, as the benchmark's developed flow has them."""
    s = CartSolver(cases.forward_facing_step_case(65, limiter=limiter, t_end=1.14))
    s.solve()
    got = [torch.from_numpy(s.state(b)[:, 2:-2, 2:-2].copy()).cuda() for b in range(s.nblocks)]
    s.close()
    return got


def _ffs_states(case, seed, spec):
    rng = np.random.default_rng(seed)
    out = []
    for b, U in enumerate(_developed(case["limiter"])):
        nx, ny = spec["mesh"]["blocks"][b]["x_cells"], spec["mesh"]["blocks"][b]["y_cells"]
        U = torch.nn.functional.interpolate(U[None], size=(ny, nx), mode="bilinear")[0]
        x, y = _grid(nx, ny)
        f, ph = rng.integers(2, 9, 2), rng.uniform(0, 2 * math.pi, 2)
        # all four conserved fields by one factor: the velocity stays, rho and p vary by a per cent
        U = U * (1 + 0.01 * torch.sin(2 * math.pi * f[0] * x + ph[0]) * torch.sin(2 * math.pi * f[1] * y + ph[1]))
        out.append(_pad(U, 2))
    return out


def _cart_case(case):
    if case["kind"] == "ffs":
        return cases.forward_facing_step_case(case["h"], limiter=case["limiter"])
    return cases.quadrant_case(case["nx"], ny=case["ny"], scheme=case["scheme"], limiter=case["limiter"] or None,
                               cfl=cases.CFL_2D)


def _cart_states(case, seed, spec):
    if case["kind"] == "ffs":
        return _ffs_states(case, seed, spec)
    x, y = _grid(case["nx"], case["ny"])
    return [_pad(_cons(*_flow(x, y, np.random.default_rng(seed))), 1 if case["scheme"] == "Godunov" else 2)]


def _sides(case):
    """The batch's sides: log-spaced from lo to hi, the odd ones among them."""
    n = case["count"]
    return [int(round(case["lo"] * (case["hi"] / case["lo"]) ** (k / max(1, n - 1)))) | (k & 1) for k in range(n)]


def _batch_specs(case):
    return [cases.quadrant_case(n, scheme=case["scheme"], limiter=case["limiter"] or None, cfl=cases.CFL_2D)
            for n in _sides(case)]


def _batch_states(case, seed):
    rng = np.random.default_rng(seed)
    return [_cons(*_flow(*_grid(n, n), rng)) for n in _sides(case)]


@functools.lru_cache(maxsize=2)
def _mesh(cells):
    """A triangle mesh of [0, 4] x [0, 2] with a rectangular hole: a jittered lattice, every square
    cut along one of its diagonals.  Returns vertices [n, 3, 2], boundary codes [n, 3] (-1 wall,
    -2 outflow, -3 inlet, 0 interior) and neighbours [n, 3] (the code at a boundary)."""
    ny = max(8, int(round(math.sqrt(cells / 4.0))))
    nx = 2 * ny
    rng = np.random.default_rng(7)
    X, Y = np.meshgrid(np.linspace(0.0, 4.0, nx + 1), np.linspace(0.0, 2.0, ny + 1))
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1))
    hole = lambda a, b: (a > 0.25 * nx) & (a < 0.35 * nx) & (b > 0.4 * ny) & (b < 0.6 * ny)  # noqa: E731
    free = (i > 0) & (i < nx) & (j > 0) & (j < ny) & ~hole(i - 1, j) & ~hole(i + 1, j) & ~hole(i, j - 1) & \
        ~hole(i, j + 1) & ~hole(i - 1, j - 1) & ~hole(i + 1, j + 1) & ~hole(i - 1, j + 1) & ~hole(i + 1, j - 1)
    X = X + np.where(free, rng.uniform(-0.25, 0.25, X.shape), 0.0) * 4.0 / nx
    Y = Y + np.where(free, rng.uniform(-0.25, 0.25, Y.shape), 0.0) * 2.0 / ny
    a, b = np.meshgrid(np.arange(nx), np.arange(ny))
    keep = ~hole(a + 0.5, b + 0.5)
    a, b = a[keep], b[keep]
    p00, p10 = b * (nx + 1) + a, b * (nx + 1) + a + 1
    p01, p11 = p00 + nx + 1, p10 + nx + 1
    d = ((a + b) & 1 == 0)[:, None]
    t0 = np.where(d, np.stack([p00, p10, p11], 1), np.stack([p00, p10, p01], 1))
    t1 = np.where(d, np.stack([p00, p11, p01], 1), np.stack([p10, p11, p01], 1))
    tri = np.stack([t0, t1], 1).reshape(-1, 3)
    P = np.stack([X.ravel(), Y.ravel()], 1)
    e0, e1 = tri, np.roll(tri, -1, 1)
    key = (np.minimum(e0, e1).astype(np.int64) * P.shape[0] + np.maximum(e0, e1)).ravel()
    order = np.argsort(key, kind="stable")
    same = key[order][1:] == key[order][:-1]
    nbr = np.full(key.size, -9, np.int64)
    first, second = order[:-1][same], order[1:][same]
    nbr[first], nbr[second] = second // 3, first // 3
    nbr = nbr.reshape(-1, 3)
    mid = 0.5 * (P[e0] + P[e1])
    code = np.where(nbr >= 0, 0, -1)
    edge = (mid[..., 0] > 4.0 - 1e-9) | (mid[..., 1] < 1e-9) | (mid[..., 1] > 2.0 - 1e-9)
    code = np.where((nbr < 0) & edge, -2, code)
    code = np.where((nbr < 0) & (mid[..., 0] < 1e-9), -3, code)
    return P[tri], code, np.where(nbr >= 0, nbr, code)


def _mesh_bytes(V, code):
    """the binary mesh format (the loader takes it as the text format's equal)"""
    n = len(V)
    head = b"HFMESHB1" + np.array([n, 3 * n], "<i8").tobytes()
    ints = np.full(n, 3, "<i4").tobytes() + code.astype("<i4").tobytes()
    return head + ints + b"\0" * (-(len(head) + len(ints)) % 8) + V.astype("<f8").tobytes()


UNS_CASE = {
    "model": {"model": "EulerIdealGas", "gamma": GAMMA},
    "mesh": {"type": "hyperflow_unstructured", "file": "", "boundaries": {"inlet": [1.4, 2.0, 0.0, 1.0]}},
    "domain": {"x_left": 0.0, "x_right": 4.0, "y_bottom": 0.0, "y_top": 2.0,
               "boundaries": [[[0.0, 0.0], [4.0, 0.0], [4.0, 2.0], [0.0, 2.0]]]},
    "initial_condition": {"type": "Constant", "variables": "Primitive", "init_state": [1.4, 2.0, 0.0, 1.0]},
    "scheme": {"type": "Godunov", "riemann": "HLLCEuler", "ode": "ForwardEuler"},
    "simulation": {"cfl": 0.5, "t_start": 0.0, "t_end": 1.0e9, "animation": {"duration": 1.0, "fps": 1.0}},
}


def _uns_state(case, seed):
    c = torch.from_numpy(_mesh(case["cells"])[0].mean(1)).cuda()
    r, u, v, p = _flow(c[:, 0] / 4.0, c[:, 1] / 2.0, np.random.default_rng(seed))
    return _cons(r, u + 1.0, v, p)


def _learned_state(n, seed):
    return _cons(*_flow(*_grid(n, n), np.random.default_rng(seed))).float()


def _max_speed(U):
    r, u, v, p = _prim(U)
    return (torch.maximum(u.abs(), v.abs()) + (GAMMA * p / r).sqrt()).max().item()


def _train_pair(case, seed):
    """(state, target, weights, dt): the target is the plain step of the state plus the smooth
    residual that a finer grid leaves."""
    n = case["n"]
    U0 = _learned_state(n, seed)
    dt = cases.CFL_2D / n / _max_speed(U0.double())
    x, y = _grid(n, n)
    T = _plain_step(U0.double(), dt * n)
    T = T * (1 + 2e-3 * torch.sin(6 * math.pi * x) * torch.sin(4 * math.pi * y))
    w = 1.0 / ((T - U0.double()) ** 2).mean(dim=(1, 2))
    return U0, T.float(), w.float(), dt


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": case}
    if kind in ("step", "run", "ffs"):
        spec = _cart_case(case)
        st["solver"] = CartSolver(spec)
        st["in"] = [_pinned(U) for U in _cart_states(case, seed, spec)]
        st["out"] = [_pinned(torch.from_numpy(U)) for U in st["in"]]
    elif kind == "batch":
        st["solver"] = BatchSolver({"cases": _batch_specs(case)})
        st["in"] = [_pinned(U) for U in _batch_states(case, seed)]
        st["solver"].autotune()
    elif kind == "uns":
        V, code, _ = _mesh(case["cells"])
        st["solver"] = UnsSolver(UNS_CASE, _mesh_bytes(V, code))
        st["solver"].set_edge_mode(case["edge"])
        st["in"] = _pinned(_uns_state(case, seed))
        st["out"] = _pinned(torch.from_numpy(st["in"]))
    else:
        n = case["n"]
        st["solver"] = LearnedSolver(n, 1.0 / n, cfl=cases.CFL_2D)
        st["params"] = init_params(seed)
        if kind == "learned":
            st["solver"].set_params(st["params"])
            U = _learned_state(n, seed)
            st["t_end"] = _learned_end(case, U)
            st["in"] = _pinned(U)
        else:
            U0, T, w, st["dt"] = _train_pair(case, seed)
            st["in"], st["target"], st["w"] = _pinned(U0), _pinned(T), w.cpu().numpy()
    return st


def _learned_end(case, U):
    # half a step past a whole number of starting steps, so that the count does not hang on a rounding
    return (case["steps"] + 0.5) * cases.CFL_2D / case["n"] / _max_speed(U.double())


def run(st):
    case, s = st["case"], st["solver"]
    kind = case["kind"]
    if kind == "ffs" and case["io"]:
        dts = [s.step_io(st["in"] if k == 0 else st["out"], st["out"]) for k in range(case["steps"])]
        return [dts, *st["out"]]
    if kind in ("step", "run", "ffs"):
        for b, U in enumerate(st["in"]):
            s.set_state(b, U)
        dts = []
        if kind == "step":
            dts = [s.step() for _ in range(case["steps"])]
        else:
            s.run(case["steps"])
        return [dts, *[s.state(b, out=o) for b, o in enumerate(st["out"])]]
    if kind == "batch":
        for i, U in enumerate(st["in"]):
            s.set_state(i, U)
        s.run(case["steps"])
        return [s.state(i) for i in range(s.ninstances)]
    if kind == "uns":
        s.set_state(st["in"])
        s.run(case["steps"])
        return s.state(out=st["out"])
    if kind == "learned":
        s.set_state(st["in"], 0.0)
        s.run_to(st["t_end"], True)
        return s.state()
    s.set_params(st["params"])
    losses = [s.train_step(st["in"], st["target"], st["w"], st["dt"], 1e-3) for _ in range(case["steps"])]
    return [losses, s.params()]


def _cells(case):
    kind = case["kind"]
    if kind in ("step", "run"):
        return case["nx"] * case["ny"]
    if kind == "ffs":
        return cases.total_cells(_cart_case(case))
    if kind == "batch":
        return sum(n * n for n in _sides(case))
    if kind == "uns":
        return len(_mesh(case["cells"])[0])
    return case["n"] ** 2


def work(case):
    """State in and out once (and the mesh's geometry); per cell and step the FP64 additions and
    multiplications of the scheme, divisions and roots counted as one each."""
    cells, steps, kind = _cells(case), case["steps"], case["kind"]
    if kind in ("learned", "train"):
        faces = 2 * case["n"] * (case["n"] + 1)
        return {"bytes": 32 * cells, "flops": steps * (16896 * faces * (3 if kind == "train" else 1) + 400 * cells)}
    if kind == "uns":
        per = 1.5 * 95 + 30 if case["edge"] else 3 * 95 + 20
        return {"bytes": (64 + 16) * cells + 60 * cells, "flops": per * cells * steps}
    per = 190 if case.get("scheme") == "Godunov" else 340
    return {"bytes": 64 * cells * (steps if case.get("io") else 1), "flops": per * cells * steps}


# --- the same results in plain 64-bit torch ------------------------------------------------------

def _prim(U):
    r, u, v = U[0], U[1] / U[0], U[2] / U[0]
    return r, u, v, (GAMMA - 1.0) * (U[3] - 0.5 * r * (u * u + v * v))


def _flux(U):
    r, u, v, p = _prim(U)
    return torch.stack([U[1], U[1] * u + p, U[1] * v, u * (U[3] + p)])


def _hllc(L, R):
    """the HLLC flux along the first momentum of two conservative states"""
    (rl, ul, vl, pl), (rr, ur, vr, pr) = _prim(L), _prim(R)
    al, ar = (GAMMA * pl / rl).sqrt(), (GAMMA * pr / rr).sqrt()
    sl, sr = torch.minimum(ul - al, ur - ar), torch.maximum(ul + al, ur + ar)
    ss = (pr - pl + rl * ul * (sl - ul) - rr * ur * (sr - ur)) / (rl * (sl - ul) - rr * (sr - ur))

    def star(U, r, u, v, p, s):
        c = r * (s - u) / (s - ss)
        us = torch.stack([c, c * ss, c * v, c * (U[3] / r + (ss - u) * (ss + p / (r * (s - u))))])
        return _flux(U) + s * (us - U)

    F = torch.where(ss >= 0, star(L, rl, ul, vl, pl, sl), star(R, rr, ur, vr, pr, sr))
    F = torch.where(sr <= 0, _flux(R), F)
    return torch.where(sl >= 0, _flux(L), F)


def _limit(r, vanleer):
    xr = 2.0 / (1.0 + r)
    x = torch.minimum(2.0 * r / (1.0 + r), xr) if vanleer else torch.where(r <= 1.0, r, xr.clamp(max=1.0))
    return torch.where(r <= 0, torch.zeros_like(r), x)


def _mh_faces(q, h, vanleer):
    """face fluxes along the last axis of q (two halo cells at either end), the first momentum normal"""
    dl, dr = q[..., 1:-1] - q[..., :-2], q[..., 2:] - q[..., 1:-1]
    clamp = lambda d: torch.where(d.abs() <= 1e-6, torch.where(d < 0, -1e-6, 1e-6).to(d), d)  # noqa: E731
    s = 0.5 * _limit(clamp(dl) / clamp(dr), vanleer) * (0.5 * dl + 0.5 * dr)
    e0, e1 = q[..., 1:-1] - s, q[..., 1:-1] + s
    d = h * (_flux(e0) - _flux(e1))
    return _hllc((e1 + d)[..., :-1], (e0 + d)[..., 1:])


def _turn(U):
    """x and y exchanged: axes and momenta"""
    return U[[0, 2, 1, 3]].transpose(1, 2).contiguous()


def _update(U, g, dt, dtp, dx, dy, scheme, vanleer):
    def along(q, h):
        return _hllc(q[..., :-1], q[..., 1:]) if scheme == "Godunov" else _mh_faces(q, h, vanleer)

    F = along(U[:, g:-g], 0.5 * dtp / dx)
    G = along(_turn(U)[:, g:-g], 0.5 * dtp / dy)
    L = (F[..., :-1] - F[..., 1:]) / dx + _turn(G[..., :-1] - G[..., 1:]) / dy
    return U[:, g:-g, g:-g] + dt * L


def _speed_dt(Us, dxy, cfl, call):
    dt = 1e16
    for U, (dx, dy) in zip(Us, dxy):
        r, u, v, p = _prim(U)
        c = (GAMMA * p / r).sqrt()
        dt = min(dt, dx / (u.abs() + c).nan_to_num(0.0).max().item(), dy / (v.abs() + c).nan_to_num(0.0).max().item())
    return (0.2 * cfl if call < 10 else cfl) * dt


def _fill(Us, spec, g):
    """the ghost cells: blocks in order, bottom, right, top, left"""
    for U, blk in zip(Us, spec["mesh"]["blocks"]):
        for side in ("bottom", "right", "top", "left"):
            bc = blk["boundaries"][side]
            ax = 1 if side in ("bottom", "top") else 2
            low = side in ("bottom", "left")
            src = Us[bc["block"]] if bc["type"] == "Internal" else U
            n, m = U.shape[ax], src.shape[ax]
            for k in range(g):
                d = g - 1 - k if low else n - g + k
                if bc["type"] == "Dirichlet":
                    w = torch.tensor(bc["flow_state"], dtype=U.dtype, device=U.device)
                    U.select(ax, d).copy_(_cons(*w)[:, None].expand_as(U.select(ax, d)))
                    continue
                if bc["type"] == "Internal":
                    at = m - g - 1 - k if low else g + k
                else:
                    at = g + k if low else n - g - 1 - k
                U.select(ax, d).copy_(src.select(ax, at))
                if bc["type"] == "Reflective":
                    U.select(ax, d)[2 if ax == 1 else 1].neg_()


def _cart_exact(Us, spec, steps):
    scheme, cfl = spec["scheme"]["type"], spec["simulation"]["cfl"]
    vanleer, g = spec["scheme"].get("limiter") == "VanLeer", 1 if scheme == "Godunov" else 2
    dxy = []
    for b in spec["mesh"]["blocks"]:
        e = b["extents"]
        dxy.append(((e["x_right"] - e["x_left"]) / b["x_cells"], (e["y_top"] - e["y_bottom"]) / b["y_cells"]))
    call, dts = 0, []
    for _ in range(steps):
        _fill(Us, spec, g)
        dt = _speed_dt(Us, dxy, cfl, call)
        call += 1
        dts.append(dt)
        for b, U in enumerate(Us):
            dtp = 0.0
            if scheme != "Godunov":   # the half-step predictor's own time step, earlier blocks updated
                dtp = _speed_dt(Us, dxy, cfl, call)
                call += 1
            U[:, g:-g, g:-g] = _update(U, g, dt, dtp, *dxy[b], scheme, vanleer)
    return dts, Us


def _uns_exact(case, seed):
    V, _, nbr = _mesh(case["cells"])
    V, nbr = torch.from_numpy(V).cuda(), torch.from_numpy(nbr).cuda()
    U = _uns_state(case, seed)
    e = torch.roll(V, -1, 1) - V
    ln = e.pow(2).sum(2).sqrt()
    nx, ny = e[..., 1] / ln, -e[..., 0] / ln
    nxt = torch.roll(V, -1, 1)
    area = 0.5 * (V[..., 0] * nxt[..., 1] - nxt[..., 0] * V[..., 1]).sum(1)
    h = ln.sum(1) / 2
    rin = (h * (h - ln[:, 0]) * (h - ln[:, 1]) * (h - ln[:, 2])).sqrt() / h
    inlet = _cons(*torch.tensor([1.4, 2.0, 0.0, 1.0], dtype=torch.float64, device="cuda"))
    for k in range(case["steps"]):
        r, u, v, p = _prim(U)
        dt = (0.1 if k < 10 else 0.5) * (rin / ((u * u + v * v).sqrt() + (GAMMA * p / r).sqrt())).min()
        acc = torch.zeros_like(U)
        for f in range(3):
            c, s, at = nx[:, f], ny[:, f], nbr[:, f]
            rot = lambda W: torch.stack([W[0], c * W[1] + s * W[2], c * W[2] - s * W[1], W[3]])  # noqa: E731
            L, R = rot(U), rot(U[:, at.clamp(min=0)])
            wall = L.clone()
            wall[1].neg_()
            R = torch.where(at == -1, wall, torch.where(at == -2, L, torch.where(at == -3, rot(inlet[:, None].expand_as(U)), R)))
            F = _hllc(L, R)
            acc += ln[:, f] * torch.stack([F[0], c * F[1] - s * F[2], s * F[1] + c * F[2], F[3]])
        U = U - dt / area * acc
    return U


def _mirror(U, g):
    U = torch.cat([U[..., :g].flip(-1), U, U[..., -g:].flip(-1)], -1)
    return torch.cat([U[..., :g, :].flip(-2), U, U[..., -g:, :].flip(-2)], -2)


def _plain_fluxes(U, r):
    q = _mirror(U, 2)
    return _mh_faces(q[:, 2:-2], 0.5 * r, False), _turn(_mh_faces(_turn(q)[:, 2:-2], 0.5 * r, False))


def _apply(U, F, G, r):
    return U + r * ((F[..., :-1] - F[..., 1:]) + (G[:, :-1] - G[:, 1:]))


def _plain_step(U, r):
    return _apply(U, *_plain_fluxes(U, r), r)


def _net(params, U):
    """the network's flux corrections on the x faces [4, n, n+1] and y faces [4, n+1, n]"""
    n = U.shape[1]
    W1, b1, W2, b2, W3, b3 = params

    def faces(W):   # along x, the first velocity normal
        q = torch.cat([W[..., :2].flip(-1), W, W[..., -2:].flip(-1)], -1)
        q = torch.cat([q[:, :1], q, q[:, -1:], q[:, -2:-1]], 1)   # tangential offsets -1 .. 2, mirrored
        rr = 0.5 * (q[0, 1:-2, 1:-2] + q[0, 1:-2, 2:-1])
        pr = 0.5 * (q[3, 1:-2, 1:-2] + q[3, 1:-2, 2:-1])
        c = (GAMMA * pr / rr).clamp(min=1e-12).sqrt()
        x = []
        for a in range(4):
            for b in range(4):
                w = q[:, b:b + n, a:a + n + 1]
                x += [w[0] / rr - 1, w[1] / c, w[2] / c, w[3] / pr - 1]
        x = torch.stack(x, -1)
        gelu = lambda z: torch.nn.functional.gelu(z, approximate="tanh")  # noqa: E731
        o = (gelu(gelu(x @ W1.T + b1) @ W2.T + b2) @ W3.T + b3).permute(2, 0, 1)
        m = rr * c
        return torch.stack([m * o[0], m * c * o[1], m * c * o[2], m * c * c * o[3]])

    W = torch.stack(_prim(U))
    return faces(W), _turn(faces(_turn(W)))


def _unpack(params):
    p, out, o = torch.from_numpy(params).cuda().double(), [], 0
    for shape in ((64, 64), (64,), (64, 64), (64,), (4, 64), (4,)):
        k = math.prod(shape)
        out.append(p[o:o + k].reshape(shape).clone())
        o += k
    return out


def _bad(un, up, u0):
    """the change guard: a non-physical state, or a density or energy change beyond half the plain one"""
    r, _, _, p = _prim(un)
    far = [(un[v] - up[v]).abs() > 0.5 * ((up[v] - u0[v]).abs() + 1e-6 * u0[v].abs()) for v in (0, 3)]
    return ~(r > 0) | ~(p > 0) | far[0] | far[1]


def _learned_exact(case, seed):
    n, net = case["n"], _unpack(init_params(seed))
    U32 = _learned_state(n, seed)
    U, t, t_end, k = U32.double(), 0.0, _learned_end(case, U32), 0
    while t < t_end:
        dt = cases.CFL_2D / n / _max_speed(U) * (0.2 if k < 5 else 1.0)
        dt = t_end - t if t + dt > t_end else dt
        F, G = _plain_fluxes(U, dt * n)
        dF, dG = _net(net, U)
        up = _apply(U, F, G, dt * n)
        bad = _bad(_apply(U, F + dF, G + dG, dt * n), up, U)
        okx, oky = torch.ones_like(F[0]), torch.ones_like(G[0])
        okx[:, :-1][bad] = 0
        okx[:, 1:][bad] = 0
        oky[:-1][bad] = 0
        oky[1:][bad] = 0
        un = _apply(U, F + okx * dF, G + oky * dG, dt * n)
        U = torch.where(_bad(un, up, U), up, un)
        t, k = t + dt, k + 1
    return U


def _train_exact(case, seed):
    U0, T, w, dt = _train_pair(case, seed)
    U, T, w, r = U0.double(), T.double(), w.double(), dt * case["n"]
    net = [p.requires_grad_() for p in _unpack(init_params(seed))]
    F, G = _plain_fluxes(U, r)
    m = [[torch.zeros_like(p) for p in net] for _ in range(2)]
    losses = []
    for k in range(1, case["steps"] + 1):
        dF, dG = _net(net, U)
        loss = (w[:, None, None] * (_apply(U, F + dF, G + dG, r) - T) ** 2).sum() / case["n"] ** 2
        grads = torch.autograd.grad(loss, net)
        losses.append(loss.item())
        with torch.no_grad():
            for p, g, a, b in zip(net, grads, *m):
                a.mul_(0.9).add_(g, alpha=0.1)
                b.mul_(0.999).addcmul_(g, g, value=0.001)
                p -= 1e-3 * (a / (1 - 0.9 ** k)) / ((b / (1 - 0.999 ** k)).sqrt() + 1e-8)
    return [losses, torch.cat([p.detach().reshape(-1) for p in net])]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "run", "ffs"):
        spec = _cart_case(case)
        dts, Us = _cart_exact(_cart_states(case, seed, spec), spec, case["steps"])
        return [dts if kind == "step" or case.get("io") else [], *Us]
    if kind == "batch":
        out = []
        g = 1 if case["scheme"] == "Godunov" else 2
        for spec, U in zip(_batch_specs(case), _batch_states(case, seed)):
            out.append(_cart_exact([_pad(U, g)], spec, case["steps"])[1][0][:, g:-g, g:-g])
        return out
    if kind == "uns":
        return _uns_exact(case, seed)
    return _learned_exact(case, seed) if kind == "learned" else _train_exact(case, seed)
