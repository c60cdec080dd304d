"""The work this framework is used for, as cases that can be timed.

A case is one call sequence through the public Python API (`Engine`,
`flock_loss`, `radix_sort_pairs`) on seeded synthetic flocks: agents uniform in
a periodic cube (optionally a share of them in Gaussian blobs), cell and search
radius 4, default launch options.  Every pass starts from the same state, so a
pass can be repeated.

  rollout   set_state, step(dt, steps), get_state: flocking of one or many
            flocks, with features, kNN lists, clustering steering or obstacles
  school    the same with the Schooling law
  crowd     one frame of the crowd sample's stage-by-stage order
  gradient  flock_loss of a rollout and its backward
  sort      the standalone stable key/value radix sort
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from behavert_b200 import Engine, params_default, radix_sort_pairs, radix_sort_scratch_bytes
from behavert_b200.autograd import flock_loss

DT = 0.1
CELL = 4.0


def _case(name, kind, flocks=1, lo=0, hi=0, neighbours=16, features=0, knn=False, clustering=False, obstacles=0,
          blobs=0.0, steps=1, mode=0, every=10, bits=0, density=1.0 / 16.0):
    c = {"kind": kind, "flocks": flocks, "lo": lo, "hi": hi, "density": density, "neighbours": neighbours, "features": features,
         "knn": knn, "clustering": clustering, "obstacles": obstacles, "blobs": blobs, "steps": steps, "mode": mode,
         "every": every, "bits": bits}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a host program that owns its agents and hands them over every frame: the smallest call
        _case("frame", "rollout", lo=4096, hi=4096),
        # the small flock of the demo over its whole run, one graph of 200 steps
        _case("rollout_small", "rollout", lo=4096, hi=4096, steps=200),
        # an ordinary simulation of odd size with longer lists
        _case("rollout_mid", "rollout", lo=100003, hi=100003, neighbours=24, steps=20),
        # the large clustered world with behaviour features: the headline workload
        _case("rollout_large", "rollout", lo=1 << 20, hi=1 << 20, neighbours=32, features=8, blobs=0.3, steps=10),
        # a parameter study: many flocks of very uneven sizes in one engine
        _case("batch", "rollout", flocks=1024, lo=128, hi=65536, steps=10),
        # topological neighbourhoods: the nearest agents kept, partly crowded world
        _case("knn", "rollout", lo=262144, hi=262144, knn=True, blobs=0.3, steps=10),
        # BehaviorClustering: steering by feature similarity, with relaxation
        _case("clustering", "rollout", lo=131072, hi=131072, features=8, clustering=True, steps=10),
        # fish schools (zones of repulsion, orientation and attraction)
        _case("schooling", "school", lo=262144, hi=262144, mode=1, steps=20),
        # an application that interleaves its own code between the stages
        _case("crowd", "crowd", lo=50000, hi=50000, neighbours=31),
        # gradients of a rollout with respect to weights and initial state
        _case("gradient", "gradient", lo=65536, hi=65536, steps=50),
        # fitting the weights of many flocks among obstacles: one iteration's loss and gradient
        _case("fitting", "gradient", flocks=64, lo=1024, hi=32768, obstacles=32, steps=40),
        # the sort on its own, as a library call
        _case("sort", "sort", lo=1000003, hi=1000003, bits=24),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["rollout", "rollout", "rollout", "batch", "school", "crowd", "gradient", "fitting", "sort"])
    neighbours = rng.randint(6, 32)
    density = math.exp(rng.uniform(math.log(0.02), math.log(0.12)))
    if kind == "rollout":
        n = _spread(rng, 500, 1 << 20)
        flavour = rng.choice(["plain", "plain", "features", "knn", "clustering"])
        return _case("", "rollout", density=density, lo=n, hi=n, neighbours=neighbours,
                     features=rng.randint(2, 12) if flavour in ("features", "clustering") else 0,
                     knn=flavour == "knn", clustering=flavour == "clustering", obstacles=rng.choice([0, 0, 16]),
                     blobs=rng.choice([0.0, 0.0, 0.3]), steps=rng.randint(1, max(1, min(100, 5_000_000 // n))))
    if kind == "batch":
        flocks, hi = _spread(rng, 4, 256), _spread(rng, 500, 30000)
        return _case("", "rollout", density=density, flocks=flocks, lo=100, hi=hi, neighbours=neighbours, steps=rng.randint(2, 10))
    if kind == "school":
        n = _spread(rng, 1000, 500000)
        return _case("", "school", density=density, lo=n, hi=n, neighbours=neighbours, mode=rng.choice([1, 2]), steps=rng.randint(1, 20))
    if kind == "crowd":
        n = _spread(rng, 1000, 300000)
        return _case("", "crowd", density=density, lo=n, hi=n, neighbours=neighbours)
    if kind == "gradient":
        n = _spread(rng, 2000, 100000)
        return _case("", "gradient", density=density, lo=n, hi=n, neighbours=neighbours, steps=rng.randint(10, 50), every=rng.randint(5, 10))
    if kind == "fitting":
        return _case("", "gradient", density=density, flocks=_spread(rng, 4, 64), lo=500, hi=_spread(rng, 2000, 20000),
                     neighbours=neighbours, obstacles=rng.randint(1, 32), steps=rng.randint(5, 30))
    n = _spread(rng, 5000, 8_000_000)
    return _case("", "sort", lo=n, hi=n, bits=rng.randint(10, 32))


def _sizes(case):
    """Agents of every flock: log-uniform in [lo, hi], the same for every seed."""
    r = np.random.default_rng(case["flocks"] + 7 * case["hi"])
    return np.round(np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["flocks"]))).astype(int).tolist()


def _side(n, density):
    return CELL * max(3, int(round((n / density) ** (1.0 / 3.0) / CELL)))


def _inputs(case, seed):
    """Flock parameters (host) and agents (GPU), from the seed alone."""
    host = random.Random(seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    sizes = _sizes(case)
    n = sum(sizes)
    sides = [_side(m, case["density"]) for m in sizes]

    def per_agent(values, dtype=torch.float32):
        v = torch.tensor(values, dtype=dtype, device="cuda")
        return torch.repeat_interleave(v, torch.tensor(sizes, device="cuda"))

    rand = lambda *shape: torch.rand(*shape, generator=gen, device="cuda")  # noqa: E731
    L = per_agent(sides)[:, None]
    xyz = rand(n, 3) * L
    if case["blobs"]:
        blobs = max(1, n // 16384)
        members = rand(n) < case["blobs"]
        centres = rand(blobs, 3) * L[:1]
        which = torch.randint(blobs, (n,), generator=gen, device="cuda")
        near = centres[which] + 6.0 * torch.randn(n, 3, generator=gen, device="cuda")
        xyz = torch.where(members[:, None], torch.remainder(near, L), xyz)
    xyz = torch.where(xyz < L, xyz, torch.zeros_like(xyz))
    pos = torch.cat([xyz, torch.ones(n, 1, device="cuda")], 1)
    head = torch.randn(n, 3, generator=gen, device="cuda")
    head = head / head.norm(dim=1, keepdim=True)
    speed = torch.full((n, 1), 3.0, device="cuda") if case["kind"] == "school" else 0.5 + 0.5 * rand(n, 1)
    fwd = torch.cat([head, speed], 1)
    feat = rand(n, case["features"]) if case["features"] else None
    params = []
    for m, side in zip(sizes, sides):
        p = params_default()
        p.numBodies, p.worldSize, p.cellSize, p.commonSearchRadius = m, side, CELL, CELL
        p.maxNeighbors, p.useKnn, p.featuresCount = case["neighbours"], int(case["knn"]), case["features"]
        weights = [host.uniform(0.5, 2.0) for _ in range(3)] if case["flocks"] > 1 else [1.5, 1.0, 1.0]
        for law, w in zip((p.separationParams, p.alignmentParams, p.cohesionParams), weights):
            law[0], law[1], law[2] = w, CELL, -2.0
        if case["features"]:
            p.featureRelaxRate = 0.05
        if case["clustering"]:
            p.clusteringForceParams[0], p.alignmentClusteringForceParams[0] = 1.0, 0.5
        if case["obstacles"]:
            p.set_obstacles([[host.uniform(0, side) for _ in range(3)] + [host.uniform(2.0, 8.0)]
                             for _ in range(case["obstacles"])])
            p.obstacleAvoidanceWeight = 2.0
        p.schooling.mode, p.schooling.seed = case["mode"], host.getrandbits(31)
        params.append(p)
    target = torch.remainder(xyz + 2.0 * torch.randn(n, 3, generator=gen, device="cuda"), L) \
        if case["kind"] == "gradient" else None
    return {"sizes": sizes, "params": params, "pos": pos, "fwd": fwd, "feat": feat, "target": target}


def prepare(case, seed):
    if case["kind"] == "sort":
        n, bits = case["lo"], case["bits"]
        gen = torch.Generator(device="cuda").manual_seed(seed)
        keys = torch.randint(1 << bits, (n,), generator=gen, device="cuda", dtype=torch.int64)
        pairs = torch.stack([keys, torch.arange(n, device="cuda")], 1)
        pairs = torch.where(pairs >= 1 << 31, pairs - (1 << 32), pairs).to(torch.int32).contiguous()
        scratch = torch.empty(radix_sort_scratch_bytes(n, bits), dtype=torch.uint8, device="cuda")
        return {"case": case, "pairs": pairs, "out": torch.empty_like(pairs), "scratch": scratch}
    s = _inputs(case, seed)
    n = s["pos"].shape[0]
    engine = Engine(s["params"])
    state = {"case": case, "engine": engine}
    if case["kind"] == "gradient":
        weights = torch.tensor([[p.separationParams[0], p.alignmentParams[0], p.cohesionParams[0]] for p in s["params"]],
                               device="cuda")
        state.update(weights=weights.requires_grad_(), pos=s["pos"][:, :3].contiguous().requires_grad_(),
                     vel=(s["fwd"][:, :3] * s["fwd"][:, 3:]).contiguous().requires_grad_(), target=s["target"])
    else:
        state.update(pos=s["pos"], fwd=s["fwd"], acc=torch.zeros(n, 4, device="cuda"), feat=s["feat"])
        # where the results go: the program's own buffers
        state["out"] = {k: torch.empty_like(v) for k, v in state.items() if k in ("pos", "fwd", "acc", "feat") and v is not None}
        stats = torch.tensor([0.0, 0.5, 1.0, 0.0], device="cuda").repeat(n, 1) if case["clustering"] else None
        state["stats"] = stats
        engine.step_prepare(DT, case["steps"])
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "sort":
        radix_sort_pairs(state["pairs"], state["out"], case["lo"], case["bits"], state["scratch"])
        return state["out"]
    engine = state["engine"]
    if case["kind"] == "gradient":
        inputs = (state["weights"], state["pos"], state["vel"])
        loss = flock_loss(engine, *inputs, state["target"], DT, case["steps"], case["every"])
        return [loss.detach(), *torch.autograd.grad(loss.sum(), inputs)]
    engine.set_state(state["pos"], state["fwd"], state["acc"], state["feat"])
    if state["stats"] is not None:
        engine.set_similarity_stats(state["stats"])
    if case["kind"] == "crowd":
        for _ in range(case["steps"]):
            engine.update_crowd(DT)
    else:
        engine.step(DT, case["steps"])
    out = state["out"]
    engine.get_state_into(out["pos"], out["fwd"], out["acc"], out.get("feat"))
    return out


def work(case):
    if case["kind"] == "sort":
        return {"bytes": 16.0 * case["lo"], "flops": 0.0}
    # a step takes an agent's state (three float4 and the features) to the next one's; of its arithmetic: the
    # distances to the agents in the 27 cells around it and the steering sums over the listed ones
    agent_steps = float(sum(_sizes(case))) * case["steps"]
    near = 27.0 * CELL ** 3 * case["density"]
    listed_ones = min(case["neighbours"], 4.0 / 3.0 * math.pi * CELL ** 3 * case["density"])
    flops = near * 9.0 + listed_ones * (40.0 + 6.0 * case["features"])
    backward = 3.0 if case["kind"] == "gradient" else 1.0
    return {"bytes": backward * agent_steps * 2.0 * (48.0 + 4.0 * case["features"]), "flops": backward * agent_steps * flops}


# ---------------------------------------------------------------------------
# The same laws in 64 bits, as plain torch.


def _per_agent(s):
    """Per-agent parameters in 64 bits, and the flock of every agent."""
    sizes = torch.tensor(s["sizes"], device="cuda")
    flock = torch.repeat_interleave(torch.arange(len(s["sizes"]), device="cuda"), sizes)
    ps = s["params"]
    G = torch.tensor([round(p.worldSize / p.cellSize) for p in ps], device="cuda")
    L = torch.tensor([p.worldSize for p in ps], dtype=torch.float64, device="cuda")
    base = torch.cumsum(G ** 3, 0) - G ** 3
    weights = torch.tensor([[p.separationParams[0], p.alignmentParams[0], p.cohesionParams[0]] for p in ps], device="cuda").double()
    return {"flock": flock, "G": G[flock], "L": L[flock][:, None], "base": base[flock], "cells": int((G ** 3).sum()),
            "weights": weights}


def _pairs(a, pos, limit):
    """(agent, neighbour, neighbour's image minus the agent) of every list: the
    27 cells x outermost and z innermost, by id inside a cell, the first
    `limit` within the radius."""
    n = pos.shape[0]
    g = torch.clamp((pos / CELL).floor().long(), min=0)
    g = torch.minimum(g, a["G"][:, None] - 1)
    key = a["base"] + (g[:, 2] * a["G"] + g[:, 1]) * a["G"] + g[:, 0]
    order = torch.argsort(key, stable=True)
    start = torch.searchsorted(key[order].contiguous(), torch.arange(a["cells"] + 1, device="cuda"))
    o = torch.tensor([[x, y, z] for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)], device="cuda")
    found = []
    for lo in range(0, n, 50000):
        i = torch.arange(lo, min(n, lo + 50000), device="cuda")
        c = g[i][:, None, :] + o[None]
        G = a["G"][i][:, None, None]
        wrap = (c < 0).long() - (c >= G).long()
        c = c + wrap * G
        cell = a["base"][i][:, None] + (c[..., 2] * G[..., 0] + c[..., 1]) * G[..., 0] + c[..., 0]
        first = start[cell]
        count = start[cell + 1] - first
        flat = torch.repeat_interleave(torch.arange(cell.numel(), device="cuda"), count.reshape(-1))
        within = torch.arange(flat.numel(), device="cuda") - (torch.cumsum(count.reshape(-1), 0) - count.reshape(-1))[flat]
        j = order[first.reshape(-1)[flat] + within]
        me = i[flat // 27]
        shift = -(wrap.reshape(-1, 3)[flat].double()) * a["L"][me]
        off = (pos[j] + shift) - pos[me]
        keep = (off.square().sum(1) <= CELL * CELL) & (j != me)
        me, j, shift = me[keep], j[keep], shift[keep]
        rank = torch.arange(me.numel(), device="cuda") - torch.searchsorted(me.contiguous(), me.contiguous())
        keep = rank < limit
        found.append((me[keep], j[keep], shift[keep]))
    return [torch.cat(x) for x in zip(*found)]


def _sum(me, terms, n):
    return torch.zeros(n, terms.shape[1], dtype=torch.float64, device="cuda").index_add(0, me, terms)


def _unit(v, where):
    out = torch.zeros_like(v)
    at = where.nonzero().flatten()
    return out.index_copy(0, at, v[at] / v[at].norm(dim=1, keepdim=True))


def _clip(v, top):
    length = v.norm(dim=1, keepdim=True)
    return torch.where(length > top, v * (top / length.clamp(min=1e-300)), v)


def _limit_turn(source, cosine, basis):
    length = source.norm(dim=1, keepdim=True)
    along = (source * basis).sum(1, keepdim=True)
    aside = source - basis * along
    sine = torch.as_tensor(1 - cosine ** 2).clamp(min=0).sqrt()
    turned = (basis * cosine + aside / aside.norm(dim=1, keepdim=True) * sine) * length
    return torch.where((length > 0) & (along / length.clamp(min=1e-300) < cosine), turned, source)


def _obstacle_force(s, a, pos):
    force = torch.zeros_like(pos)
    for k in range(s["params"][0].numObstacles):
        c = torch.tensor([list(p.obstacles[k]) for p in s["params"]], device="cuda").double()[a["flock"]]
        off = pos - c[:, :3]
        off = off - a["L"] * ((off > a["L"] / 2).double() - (off < -a["L"] / 2).double())
        d, reach = off.norm(dim=1, keepdim=True), c[:, 3:] + CELL
        force = force + torch.where((d < reach) & (d > 0), off * ((1 - d / reach) / d.clamp(min=1e-300)), torch.zeros_like(off))
    return force * s["params"][0].obstacleAvoidanceWeight


def _relax(me, j, feat, n):
    norm = feat.norm(dim=1)
    sim = ((feat[me] * feat[j]).sum(1) / (norm[me] * norm[j]) + 1) / 2
    total = _sum(me, sim[:, None], n)
    mean = _sum(me, sim[:, None] * feat[j], n) / total.clamp(min=1e-300)
    return torch.where(total > 0, feat + 0.05 * (mean - feat), feat)


def _step64(case, s, a, x, weights):
    """One step of x = (pos, fwd, speed, acc, feat)."""
    pos, fwd, speed, acc, feat = x
    n = pos.shape[0]
    with torch.no_grad():
        me, j, shift = _pairs(a, pos.detach(), case["neighbours"])
    off = (pos[j] + shift) - pos[me]
    if case["kind"] == "school":
        dist = off.norm(dim=1, keepdim=True)
        away = (dist < 1.0).flatten()
        push = -_sum(me[away], (off / dist)[away], n)
        pull = _sum(me, off / dist, n) + 16.0 * (fwd / fwd.norm(dim=1, keepdim=True) + _sum(me, fwd[j] / fwd[j].norm(dim=1, keepdim=True), n))
        alone = (torch.bincount(me[away], minlength=n) == 0)[:, None]
        turn = torch.where(alone, pull, push)
        fwd = _limit_turn(_unit(turn, turn.norm(dim=1) > 0), math.cos(0.1), fwd)
        return torch.remainder(pos + fwd * 3.0 * 0.1, a["L"]), fwd, speed, acc, feat
    count = torch.bincount(me, minlength=n)
    some, c = count > 0, count.clamp(min=1)[:, None]
    sep = _unit(_sum(me, -off / off.square().sum(1, keepdim=True), n), some) * weights[:, :1]
    if case["kind"] == "crowd":
        sep = torch.where(count[:, None] > 16, sep * ((count[:, None] - 16) * 0.5), sep)
        d = (sep * fwd).sum(1, keepdim=True)
        speed = torch.where(d < -0.8, speed * 0.9, torch.where(d > 0.5, speed * 1.02, speed))
    ali = _unit(_sum(me, fwd[j], n) / c - fwd, some) * weights[:, 1:2]
    coh = _unit(_sum(me, off, n) / c, some) * weights[:, 2:]
    force = sep + ali + coh
    if case["obstacles"]:
        force = force + _obstacle_force(s, a, pos)
    slow = ((speed.detach() <= 0.2).flatten() & (force.detach().norm(dim=1) > 0)).nonzero().flatten()
    if slow.numel():
        cosine = 1 - 2 * (speed[slow] / 0.2) ** 20
        force = force.index_copy(0, slow, _limit_turn(force[slow], cosine, fwd[slow]))
    force = _clip(force, 0.1)
    acc = acc + (force - acc) * 0.4
    v = _clip(fwd * speed + acc * DT, 1.0)
    speed = v.norm(dim=1, keepdim=True)
    if feat is not None:
        feat = _relax(me, j, feat, n)
    pos = pos + v * DT
    pos = pos - a["L"] * ((pos >= a["L"]).double() - (pos < 0).double())
    return pos, v / speed, speed, acc, feat


def exact(case, seed):
    # None: whole numbers (sort); lists with an order of their own (the reference's kNN replacement, the running
    # similarity statistics of clustering); horizons and sizes over which 64 bits take another course or too long
    if case["kind"] == "sort" or case["knn"] or case["clustering"] or case["mode"] == 2:
        return None
    if case["kind"] != "gradient" and case["steps"] > 20 or sum(_sizes(case)) * case["steps"] > 12_000_000:
        return None
    s = _inputs(case, seed)
    a = _per_agent(s)
    n = s["pos"].shape[0]
    pos, fwd, speed = s["pos"][:, :3].double(), s["fwd"][:, :3].double(), s["fwd"][:, 3:].double()
    acc = torch.zeros(n, 3, dtype=torch.float64, device="cuda")
    feat = s["feat"].double() if s["feat"] is not None else None
    weights = a["weights"]
    if case["kind"] != "gradient":
        x = (pos, fwd, speed, acc, feat)
        for _ in range(case["steps"]):
            x = _step64(case, s, a, x, weights[a["flock"]])
        pos, fwd, speed, acc, feat = x
        zero, one = torch.zeros_like(speed), torch.ones_like(speed)
        out = {"pos": torch.cat([pos, one], 1), "fwd": torch.cat([fwd, speed], 1), "acc": torch.cat([acc, zero], 1)}
        if feat is not None:
            out["feat"] = feat
        return out
    vel = (s["fwd"][:, :3] * s["fwd"][:, 3:]).double()
    inputs = [t.requires_grad_() for t in (weights, pos, vel)]
    speed = vel.norm(dim=1, keepdim=True)
    x = (pos, vel / speed, speed, acc, None)
    for _ in range(case["steps"]):
        x = _step64(case, s, a, x, weights[a["flock"]])
    d = x[0] - s["target"].double()
    d = d - a["L"] * ((d > a["L"] / 2).double() - (d < -a["L"] / 2).double())
    sizes = torch.tensor(s["sizes"], dtype=torch.float64, device="cuda")
    loss = torch.zeros(len(s["sizes"]), dtype=torch.float64, device="cuda").index_add(0, a["flock"], d.square().sum(1)) / sizes
    return [loss.detach(), *torch.autograd.grad(loss.sum(), inputs)]
