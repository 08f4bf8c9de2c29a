"""Performance cases of the delta-SPH library: what its users have it do, through the public
Python handles over the C ABI (tmp_sph_gb300.solver), with inputs made from a seed alone.

Kinds of cases:

  advance   a resident simulation: the state is uploaded from device arrays, advanced a few
            predictor-corrector steps as graph replays, and read back in original order
  batch     several independent dam breaks of uneven size advanced by one set of launches
  host      one end-to-end step on pinned host arrays (sph_step_host), the arrays advanced in place
  drop_in   one step of the reference's own step loop through the drop-in functions: hash, sort,
            reorder, both neighbour passes, predictor or corrector, recover, twice per step
  probe     gauges, pressure probes, surge front and the FP64 reductions of a resident state
  cells     the cell list alone: hash, stable sort and reorder of particles in random order

A flow is either "early" (a hydrostatic water column on a slightly jittered lattice that has
begun to move, 0.1-0.3 m/s, as in the first hundreds of steps of a dam break: neighbour lists
last for tens of steps) or "surge" (the collapsing column: an outflow of 1.2-1.8 m/s on a
disordered lattice: lists are rebuilt every few steps).  Both are divergence-free.

exact() restates the physics in 64-bit torch, without the library.
"""
from __future__ import annotations

import math

import numpy as np
import torch

G, RHO0, GAMMA = -9.81, 1000.0, 7.0
PI = 3.141592654  # as the parameter derivation of the library (and of the reference code) has it
LAYERS = 3        # wall layers of the generated tank

# ---------------------------------------------------------------- the cases


def _advance(name, dx, tank, block, *, precision="fp32", flow="early", physics="config", steps=10,
             obstacle=False):
    return dict(name=name, kind="advance", dx=dx, tx=tank[0], ty=tank[1], tz=tank[2], bx=block[0],
                by=block[1], bz=block[2], precision=precision, flow=flow, physics=physics,
                steps=steps, obstacle=obstacle)


_TANK, _BLOCK = (1.0, 0.5, 0.6), (0.4, 0.5, 0.3)


def _as(kind, case, **more):
    return {**case, "kind": kind, **more}


def listed():
    return [
        # the coarsest tank (6,767 particles): set-up runs and parameter scans, all latency
        _advance("advance_7k", 0.04, _TANK, _BLOCK, steps=20),
        # the 133,968-particle dam break with the reference's physics (linear EOS, h = 1.5 dx)
        _advance("advance_134k_linear", 0.01, _TANK, _BLOCK, physics="reference", steps=10),
        # the 765,828-particle dam break while the column collapses, in plain FP32
        _advance("advance_766k_surge", 0.005, _TANK, _BLOCK, flow="surge", steps=10),
        # the headline 4.96M-particle dam break in its first steps
        _advance("advance_5m", 0.0025, _TANK, _BLOCK, steps=5),
        # the long tank with a rigid obstacle (6.8M particles) in a developed flow: the largest
        _advance("advance_obstacle_7m", 0.005, (3.22, 1.0, 1.0), (1.2, 1.0, 0.55), flow="surge",
                 steps=5, obstacle=True),
        # mixed precision on cell-local offsets, the form for accurate long runs
        _advance("advance_766k_mixed", 0.005, _TANK, _BLOCK, precision="mixed", flow="surge",
                 steps=5),
        # the FP64 solver every accuracy study runs beside the others
        _advance("advance_134k_fp64", 0.01, _TANK, _BLOCK, precision="fp64", steps=3),
        # six uneven dam breaks in one batch, mixed precision on FP32 positions (parameter study)
        _as("batch", _advance("batch_6_mixed_abs", 0.005, _TANK, (0.6, 0.5, 0.45),
                              precision="mixed_abs", steps=5), instances=6),
        # a driver that keeps its state on the host and calls one step at a time
        _as("host", _advance("host_step_766k", 0.005, _TANK, _BLOCK, steps=1)),
        # the reference's own step loop linked against the drop-in functions
        _as("drop_in", _advance("drop_in_766k", 0.005, _TANK, _BLOCK, steps=1)),
        # the gauges a run reads every output interval, on the headline state
        _as("probe", _advance("probe_5m", 0.0025, _TANK, _BLOCK, steps=0)),
        # cell list of 2.1M particles in the order a particle file has them
        _as("cells", _advance("cells_2m", 0.007, (3.0, 1.0, 1.0), (1.0, 1.0, 0.5), steps=0)),
    ]


def draw(rng):
    """One more case of these ranges: any tank, 5,000 to 4M particles, each kind and option."""
    kind = rng.choices(["advance", "batch", "host", "drop_in", "probe", "cells"],
                       [10, 2, 2, 2, 1, 2])[0]
    precision = rng.choices(["fp32", "mixed_abs", "mixed", "mixed_comp", "fp64"],
                            [8, 3, 3, 1, 2])[0]
    if kind in ("drop_in", "cells"):
        precision = "fp32"
    if kind == "batch" and precision == "fp64":
        precision = "mixed_abs"
    most = 1.5e5 if precision == "fp64" else 1.5e6 if kind in ("drop_in", "host") else 4.0e6
    # a host loop goes on from pass to pass: large enough to stay in a dam break's first steps
    least = 5.0e3 if kind != "host" else 1.0e5
    target = math.exp(rng.uniform(math.log(least), math.log(most)))
    tank = [round(rng.uniform(0.6, 2.4), 3), round(rng.uniform(0.3, 1.0), 3),
            round(rng.uniform(0.5, 1.0), 3)]
    block = [round(rng.uniform(0.25, 0.5) * tank[0], 3), tank[1],
             round(rng.uniform(0.3, 0.6) * tank[2], 3)]
    inst = rng.randint(2, 12) if kind == "batch" else 1
    lo, hi = 1e-3, 0.1
    for _ in range(40):  # the spacing that gives about `target` particles in all
        dx = math.sqrt(lo * hi)
        lo, hi = (dx, hi) if inst * _count(dx, tank, block) > target else (lo, dx)
    dx = float("%.5g" % hi)
    steps = {"host": 1, "drop_in": 1, "probe": 0, "cells": 0}.get(kind)
    if steps is None:
        steps = max(2, min(20, int(1.5e7 / target)))
    if precision == "fp64":
        steps = min(steps, 3)
    case = _advance("", dx, tank, block, precision=precision,
                    flow="early" if kind == "host" else rng.choice(["early", "surge"]),
                    physics=rng.choices(["config", "reference"], [3, 1])[0], steps=steps)
    if kind == "batch":
        case["physics"] = "config"
        case["instances"] = inst
    del case["name"]
    case["kind"] = kind
    return case


# ---------------------------------------------------------------- inputs


def _cells(length, dx):
    return int(math.floor(length / dx + 0.5))


def _count(dx, tank, block):
    t, b = [_cells(v, dx) for v in tank], [_cells(v, dx) for v in block]
    walls = (t[0] + 2 * LAYERS) * (t[1] + 2 * LAYERS) * (t[2] + LAYERS) - t[0] * t[1] * t[2]
    return walls + b[0] * b[1] * b[2]


def _f(v):
    """v rounded to FP32, as a double."""
    return float(np.float32(v))


def _constants(case):
    """The simulation constants (FP32 values) of a case's physics."""
    dx = _f(case["dx"])
    column = 0.3
    if case["kind"] == "batch":
        column = max(b[2] for b in _blocks(case))
    if case["physics"] == "config":
        hf, cs, delta, alpha, tait = 1.3, _f(10.0 * math.sqrt(2.0 * 9.81 * column)), 0.1, 0.02, True
        dt = _f(_f(0.25) * _f(hf * dx) / cs)
    else:
        hf, cs, delta, alpha, tait = 1.5, 25.0, 0.2, 0.05, False
        dt = _f(2e-4)
        # the reference's fixed step is for dx of 1 cm and more: finer lattices take the CFL step
        if dx < 0.0099:
            dt = _f(_f(0.25) * _f(hf * dx) / cs)
    h = _f(hf * dx)
    return dict(dx=dx, h=h, kh=_f(2.0 * h), eta=_f(0.1 * h), mass=_f(dx ** 3 * RHO0),
                adh=_f(21.0 / (16.0 * PI * h * h * h)), cs=cs, delta=_f(delta), alpha=_f(alpha),
                dt=dt, g=_f(G), tait=tait, b=_f(RHO0 * cs * cs / GAMMA))


def _blocks(case):
    """The water blocks of the instances: one, or a fixed uneven set for a batch."""
    top = (case["bx"], case["by"], case["bz"])
    n = case.get("instances", 1) if case["kind"] == "batch" else 1
    if n == 1:
        return [top]
    r = np.random.RandomState(12)
    return [(top[0] * (1.0 if k == 0 else r.uniform(0.4, 1.0)), top[1],
             top[2] * (1.0 if k == 0 else r.uniform(0.4, 1.0))) for k in range(n)]


def _lattice(nx, ny, nz, off, device):
    i = torch.arange(nx, device=device) - off[0]
    j = torch.arange(ny, device=device) - off[1]
    k = torch.arange(nz, device=device) - off[2]
    kk, jj, ii = torch.meshgrid(k, j, i, indexing="ij")
    return torch.stack([ii.reshape(-1), jj.reshape(-1), kk.reshape(-1)], 1)


def _dam_break(case, block, seed, device):
    """One dam break in original order (walls, rigid obstacle, then fluid), FP32 on the GPU."""
    c = _constants(case)
    dx = c["dx"]
    gen = torch.Generator(device=device)
    gen.manual_seed(int(seed) * 7919 + 17)
    t = [_cells(case[k], dx) for k in ("tx", "ty", "tz")]
    w = _lattice(t[0] + 2 * LAYERS, t[1] + 2 * LAYERS, t[2] + LAYERS, (LAYERS,) * 3, device)
    inside = ((w[:, 0] >= 0) & (w[:, 0] < t[0]) & (w[:, 1] >= 0) & (w[:, 1] < t[1]) &
              (w[:, 2] >= 0))
    parts = [((w[~inside].double() + 0.5) * dx, 0)]
    b = [_cells(v, dx) for v in block]
    fluid = (_lattice(b[0], b[1], b[2], (0, 0, 0), device).double() + 0.5) * dx
    if case.get("obstacle"):
        box = (_lattice(t[0], t[1], t[2], (0, 0, 0), device).double() + 0.5) * dx
        lo = torch.tensor([2.32, 0.3, 0.0], device=device, dtype=torch.float64)
        hi = torch.tensor([2.48, 0.7, 0.16], device=device, dtype=torch.float64)
        parts.append((box[((box >= lo) & (box <= hi)).all(1)], 2))
    parts.append((fluid, 1))
    x = torch.cat([p for p, _ in parts])
    typ = torch.cat([torch.full((len(p),), k, device=device, dtype=torch.int32) for p, k in parts])
    n, fl = len(x), typ == 1
    surge = case["flow"] == "surge"
    jitter = (0.15 if surge else 0.01) * dx
    move = (torch.rand(n, 3, generator=gen, device=device, dtype=torch.float64) * 2 - 1) * jitter
    x = x + (torch.where(fl[:, None], move, torch.zeros_like(move)) if surge else move)
    top = (1.2, 0.6) if surge else (0.1, 0.2)
    a = (top[0] + top[1] * float(torch.rand(1, generator=gen, device=device))) / (b[0] * dx)
    v = torch.stack([a * x[:, 0], torch.zeros_like(x[:, 0]), -a * x[:, 2]], 1)
    v[~fl] = 0.0
    p = torch.where(fl, RHO0 * 9.81 * (b[2] * dx - x[:, 2]).clamp(min=0.0), 0.0)
    rho = RHO0 * (p / c["b"] + 1.0) ** (1.0 / GAMMA) if c["tait"] else RHO0 + p / c["cs"] ** 2
    return dict(pos=x.float(), vel=v.float(), rho=rho.float(), p=p.float(), type=typ)


def _inputs(case, seed, device="cuda"):
    """The state in original order and the particle offsets of its instances."""
    parts = [_dam_break(case, blk, seed * 64 + k, device) for k, blk in enumerate(_blocks(case))]
    st = parts[0] if len(parts) == 1 else {k: torch.cat([q[k] for q in parts]) for k in parts[0]}
    if case["kind"] == "cells":  # the order of a particle file: any
        gen = torch.Generator(device=device)
        gen.manual_seed(int(seed) + 5)
        at = torch.randperm(len(st["rho"]), generator=gen, device=device)
        st = {k: v[at].contiguous() for k, v in st.items()}
    return st, np.concatenate([[0], np.cumsum([len(q["rho"]) for q in parts])]).astype(np.int64)


def _params(case, n, nb):
    """The library's parameters for a case: its own derivation, this file's constants."""
    from tmp_sph_gb300 import api, cases as C
    d = C.geometry("precision", dx=case["dx"], tank=(case["tx"], case["ty"], case["tz"]),
                   block=(case["bx"], case["by"], case["bz"]), physics=case["physics"])
    cfg = C.config(d, case["physics"], n, nb)
    k = _constants(case)
    cfg.cs = k["cs"]
    cfg.dt = k["dt"]
    return api.params_derive(cfg)


def _probes(case):
    """Pressure on the floor and in the column, three height gauges, the surge front."""
    h, r = case["bz"], 1.5 * case["dx"]
    y = 0.5 * case["by"]
    return [(0, 0.25 * case["bx"], y, 0.1 * h, 0.0, 0.0), (0, 0.6 * case["bx"], y, 0.5 * h, 0.0, 0.0),
            (1, 0.2 * case["bx"], y, 0.0, r, 0.0), (1, 0.9 * case["bx"], y, 0.0, r, 0.0),
            (1, 0.5 * case["bx"], y, 0.0, r, 0.6 * h), (2, 0.0, 0.0, 0.0, 0.0, 0.0)]


_STREAM = []


def _stream():
    """The one stream of the program (the solver replays graphs on a stream of its own)."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _like(st, keys):
    return {k: torch.empty_like(st[k]) for k in keys}


STATE = ("pos", "vel", "rho", "p")


def prepare(case, seed):
    from tmp_sph_gb300 import api, solver as S
    st, off = _inputs(case, seed)
    n = len(st["rho"])
    nb = int((st["type"] != 1).sum())
    par = _params(case, n, nb)
    stream = _stream()
    state = dict(case=case, n=n, params=par, stream=stream)
    kind = case["kind"]
    if kind in ("advance", "batch", "probe", "host"):
        state["solver"] = S.Solver(par, n, precision=case["precision"])
    if kind in ("advance", "batch", "probe"):
        state["input"], state["out"] = st, _like(st, STATE)
    if kind == "batch":
        state["offsets"] = off.astype(np.int32)
    if kind == "probe":
        with torch.cuda.stream(stream):
            state["solver"].upload(st["pos"], st["vel"], st["rho"], st["p"], st["type"],
                                   stream=stream)
        state["probes"] = [api.SphProbe(*q) for q in _probes(case)]
    if kind == "host":
        # pinned host arrays, as a program that keeps its state on the host has them
        pinned = {k: torch.empty_like(v, device="cpu", pin_memory=True).copy_(v)
                  for k, v in st.items()}
        state["pinned"] = pinned
        state["host"] = {k: v.numpy() for k, v in pinned.items()}
    if kind in ("drop_in", "cells"):
        i32 = dict(dtype=torch.int32, device="cuda")
        state["input"] = st
        state["work"] = {k: v.clone() for k, v in st.items()}
        state["sorted"] = _like(st, (*STATE, "type"))
        state["hash"], state["index"] = torch.empty(n, **i32), torch.empty(n, **i32)
        state["start"] = torch.empty(par.num_cells, **i32)
        state["end"] = torch.zeros(par.num_cells, **i32)
        state["scratch"] = torch.empty(api.sort_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    if kind == "drop_in":
        state["solver"] = S.Solver(par, n)
        state["rates"] = dict(rho=torch.empty_like(st["rho"]), vel=torch.empty_like(st["vel"]),
                              div=torch.empty_like(st["rho"]))
        state["saved"] = _like(st, ("pos", "vel", "rho"))
    torch.cuda.synchronize()
    return state


def _cell_list(s, S, w):
    q, n, st = s["sorted"], s["n"], s["stream"]
    S.calc_hash(s["params"], w["pos"], s["hash"], s["index"], n, stream=st)
    S.sort_particles(s["hash"], s["index"], n, scratch=s["scratch"], stream=st)
    S.reorder(s["params"], w["pos"], w["vel"], w["rho"], w["p"], w["type"], None, q["pos"],
              q["vel"], q["rho"], q["p"], q["type"], None, s["hash"], s["index"], s["start"],
              s["end"], n, stream=st)


def run(state):
    from tmp_sph_gb300 import api, solver as S
    s, case, stream = state, state["case"], state["stream"]
    kind = case["kind"]
    with torch.cuda.stream(stream):
        if kind in ("advance", "batch"):
            sol, i = s["solver"], s["input"]
            if kind == "advance":
                sol.upload(i["pos"], i["vel"], i["rho"], i["p"], i["type"], stream=stream)
            else:  # device arrays: the C function itself (the handle's method takes host arrays)
                api.call("sph_upload_instances", sol.handle, *(api.ptr(i[k]) for k in STATE),
                         api.ptr(i["type"]), api.ptr(s["offsets"]), len(s["offsets"]) - 1, s["n"],
                         0, stream.cuda_stream)
            sol.step(case["steps"], stream=stream)
            sol.download_device(s["out"], stream=stream)
            return dict(s["out"])
        if kind == "host":
            s["solver"].step_host(s["host"], case["steps"], stream=stream)
            return {k: s["host"][k] for k in STATE}
        if kind == "probe":
            values, stats = s["solver"].probe(s["probes"], cfl=0.25, stream=stream)
            return dict(values=values, stats=stats)
        if kind == "cells":
            _cell_list(s, S, s["work"])
            return dict(hash=s["hash"], index=s["index"], start=s["start"], end=s["end"],
                        **{"sorted_" + k: v for k, v in s["sorted"].items()})
        # the reference's step loop, from the same state each time
        w, q, n, r, t, p = s["work"], s["sorted"], s["n"], s["rates"], s["saved"], s["params"]
        for k in STATE:
            w[k].copy_(s["input"][k])
        for half in (S.pc_prediction, S.pc_correction):
            _cell_list(s, S, w)
            s["solver"].ns(q["pos"], q["vel"], q["rho"], q["p"], q["type"], r["rho"], r["vel"],
                           s["start"], s["end"], n, s["hash"], r["div"], stream=stream)
            half(p, q["pos"], q["vel"], q["rho"], q["p"], r["rho"], r["vel"], s["index"],
                 t["pos"], t["vel"], t["rho"], n, q["type"], stream=stream)
            S.recover(w["pos"], w["vel"], w["rho"], w["p"], n, s["index"], w["type"], None,
                      q["pos"], q["vel"], q["rho"], q["p"], q["type"], None, stream=stream)
        return {k: w[k] for k in STATE}


def work(case):
    """The least a pass moves and computes.  A half step's two neighbour passes need the whole
    state of their neighbours, so each reads the 32-byte state once (the second also the first
    one's p', rho' and divergence, 12 bytes) and writes its result once (12; the new state and
    the saved or read step-n state, 32 + 28).  Pair counts: the lattice points of a sphere of
    radius kh around each fluid particle (73 flops a pair over both passes, 35 a particle)."""
    c = _constants(case)
    dx, t = c["dx"], (case["tx"], case["ty"], case["tz"])
    nf = n = 0
    for b in _blocks(case):
        n += _count(dx, t, b)
        nf += _cells(b[0], dx) * _cells(b[1], dx) * _cells(b[2], dx)
    kind = case["kind"]
    if kind == "probe":
        return {"bytes": 32.0 * n, "flops": 30.0 * nf}
    if kind == "cells":  # hash 20, sort 16, gather 72 a particle
        return {"bytes": 108.0 * n, "flops": 12.0 * n}
    halves = 2.0 * case["steps"]
    step = halves * n * (32 + 12 + 32 + 12 + 32 + 28)
    flops = halves * nf * (4.18879 * (c["kh"] / dx) ** 3 * 73 + 35)
    return {"bytes": step + 68.0 * n, "flops": flops}


# ---------------------------------------------------------------- the same in 64 bits


def _neighbours(x, inst, cut):
    """[n, K] neighbour indices of every point within `cut` of it, in its own instance; the point
    itself where a row is shorter."""
    n, dev = len(x), x.device
    c = torch.floor((x - x.min(0).values) / cut).long() + 1
    dim = (c.max(0).values + 2).tolist()
    c[:, 2] += inst.long() * (dim[2] + 1)
    key = (c[:, 2] * dim[1] + c[:, 1]) * dim[0] + c[:, 0]
    order = torch.argsort(key)
    skey = key[order]
    step = 200_000
    rows, widest = [], 1
    for a in range(0, n, step):
        i = torch.arange(a, min(n, a + step), device=dev)
        strips = torch.tensor([dz * dim[1] * dim[0] + dy * dim[0] for dz in (-1, 0, 1)
                               for dy in (-1, 0, 1)], device=dev)
        k = key[i][:, None] + strips[None]
        lo = torch.searchsorted(skey, (k - 1).contiguous())
        num = (torch.searchsorted(skey, (k + 2).contiguous()) - lo).reshape(-1)
        lo = lo.reshape(-1)
        own = torch.repeat_interleave(i.repeat_interleave(9), num)
        first = torch.cumsum(num, 0) - num
        at = torch.arange(len(own), device=dev) - torch.repeat_interleave(first - lo, num)
        j = order[at]
        near = ((x[own] - x[j]).square().sum(1) < cut * cut) & (own != j)
        own, j = own[near], j[near]
        cnt = torch.bincount(own - a, minlength=len(i))
        rank = torch.arange(len(own), device=dev) - (torch.cumsum(cnt, 0) - cnt)[own - a]
        m = int(cnt.max()) if len(own) else 1
        widest = max(widest, m)
        row = i.int()[:, None].repeat(1, max(m, 1))
        row[own - a, rank] = j.int()
        rows.append(row)
    full = []
    for k, row in enumerate(rows):
        a = k * step
        i = torch.arange(a, a + len(row), device=dev, dtype=torch.int32)
        full.append(torch.cat([row, i[:, None].repeat(1, widest - row.shape[1])], 1))
    return torch.cat(full)


def _half_step(c, nb, x, v, rho, p, fl):
    """Rates of a half step: (divergence-free) d rho/dt, dv/dt, and the walls' p and rho."""
    n, step = len(x), 1 << 16
    kh2, cfr = c["kh"] ** 2, -5.0 * c["adh"] / c["h"] ** 2
    damper, eta2 = RHO0 * c["cs"] * c["h"], c["eta"] ** 2
    visc, dhc = c["alpha"] * c["h"] * c["cs"] * RHO0, c["delta"] * c["h"] * c["cs"]
    p, rho, div = p.clone(), rho.clone(), torch.zeros_like(p)
    p0, rho0 = p.clone(), rho.clone()

    def pairs(a):
        i = torch.arange(a, min(n, a + step), device=x.device)
        j = nb[a:a + step].long()
        d = x[i][:, None] - x[j]
        r2 = d.square().sum(2)
        t = 1.0 - 0.5 * torch.sqrt(r2) / c["h"]
        return i, j, d, r2, t, (r2 < kh2) & (j != i[:, None])

    for a in range(0, n, step):
        i, j, d, r2, t, near = pairs(a)
        fj = near & fl[j]
        w = torch.where(fj, c["adh"] * t ** 4 * (5.0 - 4.0 * t), 0.0)  # 2q + 1 = 5 - 4t
        ps = ((p0[j] + rho0[j] * c["g"] * d[..., 2]) * w).sum(1)
        ws = w.sum(1)
        pw = torch.where(ws > 1e-8, ps / torch.where(ws > 1e-8, ws, 1.0), 0.0).clamp(min=0.0)
        if c["tait"]:
            rw = RHO0 * torch.expm1(torch.log1p(pw / c["b"]) / GAMMA) + RHO0
        else:
            rw = pw / c["cs"] ** 2 + RHO0
        vr = ((v[i][:, None] - v[j]) * d).sum(2)
        dv = torch.where(fj, -cfr * t ** 3 * vr * c["mass"] / rho0[j], 0.0).sum(1)
        f = fl[i]
        p[i], rho[i] = torch.where(f, p0[i], pw), torch.where(f, rho0[i], rw)
        div[i] = torch.where(f, dv, 0.0)
    drho, acc = torch.zeros_like(p), torch.zeros_like(x)
    for a in range(0, n, step):
        i, j, d, r2, t, near = pairs(a)
        w = torch.where(near, cfr * c["mass"] * t ** 3 / rho[j], 0.0)
        vr = ((v[i][:, None] - v[j]) * d).sum(2)
        inv = 1.0 / (r2 + eta2)
        drho[i] = (w * (rho[i][:, None] * vr + (rho[i][:, None] - rho[j]) * dhc * r2 * inv)).sum(1)
        s = -p[i][:, None] - p[j] + torch.where(
            fl[j], visc * vr * inv + damper * (div[i][:, None] + div[j]), 0.0)
        acc[i] = ((w * s)[..., None] * d).sum(1) / rho[i][:, None]
    acc[:, 2] += c["g"]
    return drho, acc, p, rho


def _exact_steps(case, seed):
    c = _constants(case)
    st, off = _inputs(case, seed)
    x, v, rho, p = (st[k].double() for k in STATE)
    fl = st["type"] == 1
    inst = torch.zeros(len(x), device=x.device)
    for b in range(len(off) - 1):
        inst[off[b]:off[b + 1]] = b
    nb = _neighbours(x, inst, 1.1 * c["kh"])

    def pressure(r):
        if c["tait"]:
            return c["b"] * torch.expm1(GAMMA * torch.log1p((r - RHO0) / RHO0))
        return c["cs"] ** 2 * (r - RHO0)

    hdt, f3 = 0.5 * c["dt"], fl[:, None]
    for _ in range(case["steps"]):
        drho, a, pw, rw = _half_step(c, nb, x, v, rho, p, fl)
        xn, vn, rn = x, v, rho
        rho = torch.where(fl, (rho + drho * hdt).clamp(min=RHO0), rw)
        p = torch.where(fl, pressure(rho.clamp(min=RHO0)), pw)
        x, v = torch.where(f3, x + v * hdt, x), torch.where(f3, v + a * hdt, v)
        drho, a, pw, rw = _half_step(c, nb, x, v, rho, p, fl)
        rs = (rn + drho * hdt).clamp(min=RHO0)
        rho = torch.where(fl, (2.0 * rs - rn).clamp(min=RHO0), rw)
        p = torch.where(fl, pressure(rho.clamp(min=RHO0)), pw)
        x = torch.where(f3, 2.0 * (xn + v * hdt) - xn, x)
        v = torch.where(f3, 2.0 * (vn + a * hdt) - vn, v)
    return dict(pos=x, vel=v, rho=rho, p=p)


def _exact_probe(case, seed):
    c = _constants(case)
    st, _ = _inputs(case, seed)
    f = st["type"] == 1
    x, v, rho, p = (st[k][f].double() for k in STATE)
    values = []
    for kind, px, py, pz, r, zmax in _probes(case):
        q, r = torch.tensor([_f(px), _f(py), _f(pz)], device=x.device, dtype=x.dtype), _f(r)
        if kind == 0:
            s = (x - q).square().sum(1).sqrt() / c["h"]
            w = torch.where(s < 2.0, (1.0 - 0.5 * s) ** 4 * (2.0 * s + 1.0), 0.0)
            values.append(float((p * w).sum() / w.sum()) if float(w.sum()) else 0.0)
        elif kind == 1:
            near = ((x[:, 0] - q[0]).abs() < r) & ((x[:, 1] - q[1]).abs() < r)
            if zmax > 0:
                near &= x[:, 2] < _f(zmax)
            values.append(float(x[near, 2].max()) if bool(near.any()) else 0.0)
        else:
            values.append(float(x[:, 0].max()))
    v2 = v.square().sum(1)
    top = float(v2.max().sqrt())
    stats = dict(fluid=None, parked=None, mass=c["mass"] * len(x),
                 kinetic=float(0.5 * c["mass"] * v2.sum()),
                 potential=float(-c["mass"] * c["g"] * x[:, 2].sum()), max_speed=top,
                 rho_min=float(rho.min()), rho_max=float(rho.max()), front_x=float(x[:, 0].max()),
                 cfl_dt=0.25 * c["h"] / (c["cs"] + top))
    return dict(values=values, stats=stats)


def exact(case, seed):
    if case["kind"] == "cells":
        return None  # whole numbers and copies of the input
    if case["kind"] == "probe":
        return _exact_probe(case, seed)
    return _exact_steps(case, seed)
