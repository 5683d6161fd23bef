"""Performance cases: the work a user of this framework has it do, through its public entry points.

Whole simulation steps (flamegpu2_gb300.sim.Simulation) of the bundled models from the smallest population to the
largest configuration, a batched ensemble (flamegpu2_gb300.sim.Ensemble), and the message build and the agent sort
through the kernel library's C ABI (flamegpu2_gb300.capi). A case is a dict of plain values; `prepare` makes what a
program holds before the call, `run` is one pass, `work` what the pass cannot do without, `exact` the result in 64 bits.

A simulation's pass restores the population, steps, and reads the population back. `synchronize` ends it where no
host read does: it is the call that raises the device's errors, so a program makes it before it uses the result.
"""
import ctypes as C
import math

import numpy as np
import torch

from flamegpu2_gb300 import capi, sim, synth

# The Boids configuration's weights (min_pos, max_pos and interaction_radius come from the case).
BOIDS = {"separation_radius": 0.5, "time_scale": 0.05, "global_scale": 0.15, "steer_scale": 0.005,
         "collision_scale": 0.01, "match_scale": 0.03}
F3 = ("x", "y", "z", "fx", "fy", "fz")


def listed():
    return [
        # The benchmark configuration: 16,384 Boids, 32^3 bins, wrapped, ten steps, with the population set from and
        # read back to page-locked host buffers.
        {"name": "boids_16k_host", "kind": "boids", "n": 16384, "radius": 2.0, "cells": 32, "edge": 64.0, "wrap": True,
         "steps": 10, "host": True},
        # The smallest interactive use: a thousand agents, one step, host data in and out; launches and waits count.
        {"name": "boids_1k_step", "kind": "boids", "n": 1021, "radius": 1.5, "cells": 10, "edge": 15.0, "wrap": False,
         "steps": 1, "host": True},
        # An ordinary run with the reference's default (clamped) search, a ragged population and a domain that is not
        # a whole number of radii; device-resident populations.
        {"name": "boids_100k_clamped", "kind": "boids", "n": 100003, "radius": 1.7, "cells": 47, "edge": 79.0,
         "wrap": False, "steps": 5, "host": False},
        # The ensemble configuration's largest instance: 1,048,576 Boids at one agent per bin, wrapped.
        {"name": "boids_1m", "kind": "boids", "n": 1048576, "radius": 2.5, "cells": 102, "edge": 255.0, "wrap": True,
         "steps": 1, "host": False},
        # The served request mix's second model: two agent types, 2D messages, deaths and births every step.
        {"name": "predprey_200k", "kind": "predprey", "n": 200001, "steps": 10},
        # Birth/death compaction at the benchmark's population (44-byte agents); the population falls by 16% a step.
        {"name": "birth_death_1m", "kind": "birth_death", "n": 1048576, "steps": 10},
        # The large uniform 2D configuration: 16,777,216 agents, 1024^2 bins, four payload values; the first step sorts
        # agents that come in no order, the later ones find them in bin order.
        {"name": "payload_2d_16m", "kind": "payload", "dims": 2, "n": 16777216, "steps": 5},
        # The large uneven 3D configuration: 8,388,608 agents in a 16-component Gaussian mixture on 256^3 bins.
        {"name": "payload_3d_8m", "kind": "payload", "dims": 3, "n": 8388608, "steps": 1},
        # A batched ensemble of uneven Boids instances, 100 steps, host populations in the plans, results read back.
        {"name": "ensemble_24", "kind": "ensemble", "count": 24, "hi": 65536, "steps": 100},
        # The message build alone, for a caller with its own data: unsorted input, records of an odd number of words.
        {"name": "build_3d_4m", "kind": "build", "dims": 3, "n": 4000037, "per_bin": 2.0, "words": 4,
         "order": "random", "optional": False},
        # The agent sort alone: agents that have drifted out of the last sort's order, columns of 1, 4 and 8 bytes.
        {"name": "sort_3d_2m", "kind": "sort", "dims": 3, "n": 2000003, "per_bin": 1.0, "order": "drifted"},
        # Brute-force messages, part of them not output: every agent reads every message.
        {"name": "bruteforce_16k", "kind": "bruteforce", "n": 16384, "optional": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["boids", "boids", "boids", "predprey", "birth_death", "payload", "payload", "ensemble", "build",
                       "build", "sort", "sort", "bruteforce"])
    if kind == "boids":
        n, radius, wrap = _log(rng, 1000, 1 << 20), round(rng.uniform(1.0, 4.0), 2), rng.random() < 0.5
        cells = max(3, math.ceil(rng.uniform(0.9, 1.3) * n ** (1.0 / 3.0)))
        edge = float(np.float32(np.float32(radius) * np.float32(cells)))
        if not wrap:  # the clamped search takes any domain
            edge = round(edge - rng.uniform(0.0, 0.9) * radius, 3)
        steps = rng.randint(1, 10) if n < 200000 else 1
        return {"kind": kind, "n": n, "radius": radius, "cells": cells, "edge": edge, "wrap": wrap, "steps": steps,
                "host": n < 65536 and rng.random() < 0.5}
    if kind == "predprey":
        return {"kind": kind, "n": _log(rng, 1024, 1 << 20), "steps": rng.randint(3, 12)}
    if kind == "birth_death":
        return {"kind": kind, "n": _log(rng, 1000, 1 << 20), "steps": rng.randint(2, 12)}
    if kind == "payload":
        dims = rng.choice([2, 3])
        return {"kind": kind, "dims": dims, "n": _log(rng, 1 << 15, 16000000 if dims == 2 else 3000000),
                "steps": rng.randint(1, 4)}
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(3, 24), "hi": _log(rng, 4096, 65536), "steps": rng.randint(20, 100)}
    if kind == "build":
        return {"kind": kind, "dims": rng.choice([2, 3]), "n": _log(rng, 1000, 8000000),
                "per_bin": round(rng.uniform(0.5, 24.0), 2), "words": rng.randint(0, 9),
                "order": rng.choice(["random", "drifted", "sorted"]), "optional": rng.random() < 0.3}
    if kind == "sort":
        return {"kind": kind, "dims": rng.choice([2, 3]), "n": _log(rng, 1000, 8000000),
                "per_bin": round(rng.uniform(0.5, 16.0), 2), "order": rng.choice(["random", "drifted", "sorted"])}
    return {"kind": "bruteforce", "n": _log(rng, 300, 24000), "optional": rng.random() < 0.5}


# ------------------------------------------------------------------- inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62))
    return g


def _uniform(g, n, lo, hi):
    """n float32 values in [lo, hi)."""
    t = torch.rand(n, device="cuda", generator=g, dtype=torch.float32).mul_(hi - lo).add_(lo)
    return t.clamp_(max=float(np.nextafter(np.float32(hi), np.float32(lo))))


def _ids(n):
    return torch.arange(1, n + 1, dtype=torch.int32, device="cuda")


def _boids_columns(case, seed):
    g, n = _generator(seed), case["n"]
    cols = {"_id": _ids(n)}
    for k in F3[:3]:
        cols[k] = _uniform(g, n, 0.0, case["edge"])
    for k in F3[3:]:
        cols[k] = _uniform(g, n, -1.0, 1.0)
    return cols


def _payload_shape(case):
    """Domain edge and radius of the large payload configurations at the case's population and their density."""
    if case["dims"] == 2:
        return float(np.float32(4.0 * math.sqrt(case["n"] / 16.0))), 4.0
    return float(math.ceil(256.0 * (case["n"] / float(1 << 23)) ** (1.0 / 3.0))), 1.0


def _payload_columns(case, seed):
    g, n, dims = _generator(seed), case["n"], case["dims"]
    edge, _ = _payload_shape(case)
    cols = {"_id": _ids(n)}
    if dims == 2:
        for k in ("x", "y"):
            cols[k] = _uniform(g, n, 0.0, edge)
    else:
        which = torch.randint(0, 16, (n,), device="cuda", generator=g)
        hi = float(np.nextafter(np.float32(edge), np.float32(0)))
        for k in ("x", "y", "z"):
            centre = _uniform(g, 16, 0.0, edge)
            cols[k] = (centre[which] + 2.0 * torch.randn(n, device="cuda", generator=g)).clamp_(0.0, hi)
    for k in range(4):
        cols[f"p{k}"] = _uniform(g, n, 0.0, 1.0)
    return cols


def _cells(case):
    return max(3, math.ceil((case["n"] / case["per_bin"]) ** (1.0 / case["dims"])))


def _points(case, seed, radius=1.5):
    """Positions for the build and sort cases: uniform, in no order, in bin order, or in the order of a sort that
    they have since drifted from (a twentieth of a bin)."""
    g, n, dims, cells = _generator(seed), case["n"], case["dims"], _cells(case)
    edge = cells * radius
    pos = [_uniform(g, n, 0.0, edge) for _ in range(dims)]
    if case["order"] != "random":
        key = torch.zeros(n, dtype=torch.int64, device="cuda")
        for p in reversed(pos):
            key = key * cells + (p / radius).floor().long().clamp_(0, cells - 1)
        order = torch.argsort(key, stable=True)
        pos = [p[order] for p in pos]
    if case["order"] == "drifted":
        hi = float(np.nextafter(np.float32(edge), np.float32(0)))
        pos = [(p + 0.05 * radius * torch.randn(n, device="cuda", generator=g)).clamp_(0.0, hi) for p in pos]
    return [p.contiguous() for p in pos], edge, radius, g


def _pinned(t):
    """The column in page-locked host memory, as numpy."""
    return t.cpu().pin_memory().numpy()


def _boids_params(case):
    c = dict(BOIDS, min_pos=0.0, max_pos=case["edge"], interaction_radius=case["radius"], wrap=int(case["wrap"]),
             sort_period=1)
    return synth.boids_params(c)


def prepare(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    st = {"kind": kind, "case": case}
    if kind == "boids":
        cols = _boids_columns(case, seed)
        st["sim"] = sim.Simulation("boids_spatial3d", _boids_params(case))
        if case["host"]:
            st["in"] = {k: _pinned(v).view(np.uint32 if k == "_id" else np.float32) for k, v in cols.items()}
            st["out"] = {k: _pinned(torch.empty_like(v)).view(st["in"][k].dtype) for k, v in cols.items()}
        else:
            st["pops"] = {"Boid": (cols, {k: torch.empty_like(v) for k, v in cols.items()})}
    elif kind == "payload":
        cols = _payload_columns(case, seed)
        edge, radius = _payload_shape(case)
        st["sim"] = sim.Simulation("spatial_payload", [case["dims"], 0.0, edge, radius])
        st["pops"] = {"agent": (cols, {k: torch.empty_like(v) for k, v in cols.items()})}
    elif kind == "birth_death":
        g = _generator(seed)
        cols = {"_id": _ids(n), "counter": torch.zeros(n, dtype=torch.int32, device="cuda")}
        for k in range(8):
            cols[f"f{k}"] = _uniform(g, n, 0.0, 1.0)
        st["sim"] = sim.Simulation("birth_death", [0.30, 0.20, int(seed)])
        st["pops"] = {"agent": (cols, {k: torch.zeros(2 * n, dtype=v.dtype, device="cuda") for k, v in cols.items()})}
    elif kind == "predprey":
        # three agents per unit area, a quarter of them predators, as the served requests have it
        g, n_pred = _generator(seed), max(1, n // 4)
        n_prey, edge = n - n_pred, float(math.ceil(math.sqrt(n / 3.0)))
        prey = {"_id": _ids(n_prey), "x": _uniform(g, n_prey, 0.0, edge), "y": _uniform(g, n_prey, 0.0, edge),
                "crowd": torch.zeros(n_prey, dtype=torch.int32, device="cuda")}
        pred = {"_id": _ids(n_pred), "x": _uniform(g, n_pred, 0.0, edge), "y": _uniform(g, n_pred, 0.0, edge)}
        st["sim"] = sim.Simulation("predprey2d", [edge, 1.0, 0.05, 0.02, 0.5, int(seed)])
        st["pops"] = {a: (cols, {k: torch.zeros(2 * n, dtype=v.dtype, device="cuda") for k, v in cols.items()})
                      for a, cols in (("prey", prey), ("predator", pred))}
    elif kind == "bruteforce":
        g = _generator(seed)
        cols = {"_id": _ids(n), "x": torch.randint(-50, 50, (n,), device="cuda", generator=g, dtype=torch.int32),
                "do_output": torch.ones(n, dtype=torch.int32, device="cuda"),
                "sum": torch.zeros(n, dtype=torch.int32, device="cuda"),
                "count": torch.zeros(n, dtype=torch.int32, device="cuda")}
        if case["optional"]:
            cols["do_output"] = (torch.rand(n, device="cuda", generator=g) < 0.7).to(torch.int32)
        st["sim"] = sim.Simulation("bruteforce_count", [int(case["optional"])])
        st["pops"] = {"agent": (cols, {k: torch.empty_like(v) for k, v in cols.items()})}
    elif kind == "ensemble":
        specs = synth.ensemble_instances(case["count"], n_lo=1024, n_hi=case["hi"])
        ens = sim.Ensemble("boids_spatial3d", synth.boids_params(dict(synth.BOIDS_SMALL)))
        for sp in specs:
            pop = synth.boids_population(sp["n"], 0.0, sp["edge"], int(seed) % (1 << 30) * 64 + len(specs) + ens.runs)
            r = ens.add_run(case["steps"], sp["seed"], "Boid", sp["n"], pop, "location", (0.0, 0.0, 0.0),
                            (sp["edge"],) * 3, sp["radius"])
            ens.set_property(r, "MIN_POSITION", 0.0)
            ens.set_property(r, "MAX_POSITION", sp["edge"])
            ens.set_property(r, "INTERACTION_RADIUS", sp["radius"])
        st["ens"] = ens
    elif kind == "build":
        pos, edge, radius, g = _points(case, seed)
        dims = case["dims"]
        grid = capi.grid(dims, (0.0,) * dims, (edge,) * dims, radius)
        cols = list(pos)
        if case["words"]:
            cols.append(torch.randint(0, 1 << 30, (n, case["words"]), device="cuda", generator=g, dtype=torch.int32))
        valid = (torch.rand(n, device="cuda", generator=g) < 0.8).to(torch.int32) if case["optional"] else None
        rec = capi.record_desc(cols)
        st.update(grid=grid, cols=cols, valid=valid, rec=rec,
                  sorted=torch.zeros((n, rec.words), dtype=torch.int32, device="cuda"),
                  pbm=torch.zeros(grid.binCount + 1, dtype=torch.int32, device="cuda"),
                  ws=capi.Workspace(capi.lib().fg_spatial_build_workspace_size(n, grid.binCount)))
    elif kind == "sort":
        pos, edge, radius, g = _points(case, seed)
        dims = case["dims"]
        grid = capi.grid(dims, (0.0,) * dims, (edge,) * dims, radius)
        ins = list(pos) + [_uniform(g, n, -1.0, 1.0) for _ in range(3)]
        ins += [_ids(n), torch.randint(0, 1 << 60, (n,), device="cuda", generator=g, dtype=torch.int64),
                torch.randint(0, 255, (n,), device="cuda", generator=g, dtype=torch.uint8)]
        outs = [torch.empty_like(c) for c in ins]
        st.update(grid=grid, ins=ins, outs=outs, columns=capi.columns(list(zip(ins, outs))),
                  perm=torch.empty(n, dtype=torch.int32, device="cuda"),
                  ws=capi.Workspace(capi.lib().fg_spatial_sort_workspace_size(n, C.byref(grid))))
    return st


# --------------------------------------------------------------------- pass

def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "ensemble":
        ens = state["ens"]
        if ens.simulate() != 0:
            raise RuntimeError("a run of the ensemble failed")
        return {k: np.concatenate([ens.get(r, "Boid", k, np.uint32 if k == "_id" else np.float32)
                                   for r in range(ens.runs)]) for k in ("_id",) + F3}
    if kind == "build":
        L, grid, cols = capi.lib(), state["grid"], state["cols"]
        capi.check(L.fg_spatial_build(C.byref(grid), case["n"], None, cols[0].data_ptr(), cols[1].data_ptr(),
                                      cols[2].data_ptr() if case["dims"] == 3 else None, capi.ptr(state["valid"]),
                                      C.byref(state["rec"]), state["sorted"].data_ptr(), state["pbm"].data_ptr(),
                                      state["ws"].ptr, state["ws"].nbytes, capi.stream_handle()), "fg_spatial_build")
        return {"sorted": state["sorted"], "pbm": state["pbm"]}
    if kind == "sort":
        L, grid, ins = capi.lib(), state["grid"], state["ins"]
        capi.check(L.fg_spatial_sort_agents(C.byref(grid), case["n"], None, ins[0].data_ptr(), ins[1].data_ptr(),
                                            ins[2].data_ptr() if case["dims"] == 3 else None, state["columns"],
                                            len(ins), state["perm"].data_ptr(), state["ws"].ptr, state["ws"].nbytes,
                                            capi.stream_handle()), "fg_spatial_sort_agents")
        return {"columns": state["outs"], "perm": state["perm"]}
    s = state["sim"]
    if "in" in state:  # host data in and out
        s.set_population("Boid", case["n"], state["in"])
        s.step(case["steps"])
        s.get_population("Boid", state["out"])
        return state["out"]
    for agent, (cols, _) in state["pops"].items():
        m = cols["_id"].numel()
        s.reset_population_device(agent, m, cols, m + 1)
    s.step(case.get("steps", 1))
    res = {}
    for agent, (cols, outs) in state["pops"].items():
        res[agent] = outs
        m = cols["_id"].numel()
        if kind in ("birth_death", "predprey"):  # the buffers have room for twice the population
            m = res[agent + " count"] = s.count(agent)
        for k, v in outs.items():
            s.get_device(agent, k, v[:m])
    s.synchronize()
    return res


# --------------------------------------------------------------------- work

def work(case):
    """Bytes: every agent variable, message field and index entry that a stage of the pass needs, read once and
    written once per step. Operations: the distance tests of the candidate pairs (and the sums of those in range)."""
    kind, n, steps = case["kind"], case.get("n", 0), case.get("steps", 1)
    if kind == "boids":
        bins = case["cells"] ** 3
        pairs = 27.0 * n * n / bins
        # population in and out; per step: messages written, sorted and read (28 B), PBM, agents moved and updated
        return {"bytes": 56 * n + steps * (136 * n + 8 * bins), "flops": steps * (9 * pairs + 12 * 0.155 * pairs)}
    if kind == "payload":
        dims = case["dims"]
        edge, radius = _payload_shape(case)
        bins = math.ceil(edge / radius) ** dims
        row, agent = 4 * dims + 16, 4 * dims + 20
        if dims == 2:
            pairs = 9.0 * n * n / bins
        else:  # 16 Gaussian blobs of n/16 agents, sigma 2: mean density n/16 / (8 pi^(3/2) sigma^3) over 27 unit bins
            pairs = 27.0 * n * (n / 16.0) / (8 * math.pi ** 1.5 * 8.0)
        inside = 0.349 if dims == 2 else 0.155
        return {"bytes": 2 * n * agent + steps * (4 * n * row + 2 * n * agent + 16 * n + 8 * bins),
                "flops": steps * ((3 * dims) * pairs + 5 * inside * pairs)}
    if kind == "birth_death":
        total = sum(n * 0.84 ** t for t in range(steps))
        return {"bytes": 88 * n + total * (44 + 8) + total * 0.84 * 44, "flops": 2 * total}
    if kind == "predprey":
        # prey 16 B, predators 12 B, messages 12 B; prey read both lists (9 bins at 2.25 and 0.75 per bin)
        return {"bytes": 30 * n + steps * 110 * n, "flops": steps * 0.75 * n * 27 * 5}
    if kind == "ensemble":
        # log-uniform populations in [1024, hi]
        total = case["count"] * (case["hi"] - 1024) / math.log(case["hi"] / 1024.0)
        return {"bytes": 56 * total + steps * 144 * total, "flops": steps * 27 * total * 11}
    if kind == "build":
        row = 4 * (case["dims"] + case["words"])
        words = (case["dims"] + case["words"] + 3) // 4 * 16
        return {"bytes": n * (row + words) + 4 * _cells(case) ** case["dims"], "flops": 2 * case["dims"] * n}
    if kind == "sort":
        row = 4 * case["dims"] + 12 + 4 + 8 + 1
        return {"bytes": n * (2 * row + 4), "flops": 3 * case["dims"] * n}
    return {"bytes": 60 * n, "flops": 2.0 * n * n * (0.7 if case["optional"] else 1.0)}


# -------------------------------------------------------------------- exact

def _neighbours(cells, dims, counts, start, wrap, cell, passes):
    """Yields (agents, messages) index pairs covering every message in the Moore neighbourhood of every agent, as
    rows of the bin-sorted list; None first if that takes more than `passes` row visits."""
    dev = cell[0].device
    n = cell[0].numel()
    tables = []
    for o in range(3 ** dims):
        off = [(o // 3 ** a) % 3 - 1 for a in range(dims)]
        ok = torch.ones(n, dtype=torch.bool, device=dev)
        key = torch.zeros(n, dtype=torch.int64, device=dev)
        for a in reversed(range(dims)):
            c = cell[a] + off[a]
            if wrap:
                c = c % cells
            else:
                ok &= (c >= 0) & (c < cells)
                c = c.clamp(0, cells - 1)
            key = key * cells + c
        tables.append((start[key], torch.where(ok, counts[key], torch.zeros_like(key))))
        passes -= int(tables[-1][1].sum())
        if passes < 0:
            yield None
            return
    for first, count in tables:
        rows = torch.nonzero(count > 0).reshape(-1)
        j = 0
        while rows.numel():
            yield rows, first[rows] + j
            j += 1
            rows = rows[count[rows] > j]


def _binned(pos, radius, cells):
    """Cells of float32 positions (clamped), their keys, and the bin-sorted order, counts and starts."""
    r = torch.tensor(radius, dtype=torch.float32, device="cuda")
    cell = [(p / r).floor().long().clamp_(0, cells - 1) for p in pos]
    key = torch.zeros_like(cell[0])
    for c in reversed(cell):
        key = key * cells + c
    order = torch.argsort(key, stable=True)
    counts = torch.bincount(key, minlength=cells ** len(pos))
    return [c[order] for c in cell], order, counts, torch.cumsum(counts, 0) - counts


def _sort_order(pos, edge, cells):
    """Row order after the automatic agent sort: stable by floor(p / width * cells), in float32."""
    e = torch.tensor(edge, dtype=torch.float32, device="cuda")
    key = torch.zeros(pos[0].numel(), dtype=torch.int64, device="cuda")
    for p in reversed(pos):
        key = key * cells + ((p / e) * float(cells)).floor().long()
    return torch.argsort(key, stable=True)


def _f32(v):
    return float(np.float32(v))


def exact(case, seed):
    """One step of a Boids population, or any number of a payload population's (its agents don't move), in 64 bits.
    Other runs of several steps have no such value: an agent near a bin's or a search radius's edge falls on either
    side of it, and the row order and every later step follow."""
    if case["kind"] == "boids" and case["steps"] == 1:
        out = _exact_boids(case, _boids_columns(case, seed))
        if out is None:
            return None
        out = {k: v.cpu().numpy() for k, v in out.items()} if case["host"] else out
        out["_id"] = None
        return out if case["host"] else {"Boid": out}
    if case["kind"] == "payload":
        out = _exact_payload(case, _payload_columns(case, seed))
        return None if out is None else {"agent": dict(out, _id=None)}
    return None


def _exact_boids(case, cols):
    cells, edge, wrap = int(math.ceil(np.float32(case["edge"]) / np.float32(case["radius"]))), case["edge"], case["wrap"]
    radius, sep_r = _f32(case["radius"]), _f32(BOIDS["separation_radius"])
    pos32 = [cols[k] for k in F3[:3]]
    cell, order, counts, start = _binned(pos32, case["radius"], cells)
    pos = [p.double()[order] for p in pos32]
    vel = [cols[k].double()[order] for k in F3[3:]]
    n = case["n"]
    zero = lambda: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
    centre, flow, change, seen = [zero() for _ in range(3)], [zero() for _ in range(3)], [zero() for _ in range(3)], zero()
    width = _f32(edge)
    for pair in _neighbours(cells, 3, counts, start, wrap, cell, 2_000_000_000):
        if pair is None:
            return None
        a, m = pair
        other = a != m
        a, m = a[other], m[other]
        q = []
        for k in range(3):
            d = pos[k][m] - pos[k][a]
            p = pos[k][m]
            if wrap:
                p = torch.where(d.abs() > width / 2, p - torch.sign(d) * width, p)
            q.append(p)
        dist = torch.sqrt(sum((pos[k][a] - q[k]) ** 2 for k in range(3)))
        inside = (dist < radius).double()
        close = (dist < sep_r).double() * inside * (1.0 - dist / sep_r) ** 2 * _f32(BOIDS["collision_scale"])
        seen[a] += inside
        for k in range(3):
            centre[k][a] += inside * q[k]
            flow[k][a] += inside * vel[k][m]
            change[k][a] += close * (pos[k][a] - q[k])
    have = seen > 0
    per = torch.where(have, seen, torch.ones_like(seen))
    new_v, new_p = [], []
    for k in range(3):
        steer = (centre[k] / per - pos[k]) * _f32(BOIDS["steer_scale"])
        match = flow[k] / per * _f32(BOIDS["match_scale"])
        change[k] = change[k] + torch.where(have, steer + match - vel[k], torch.zeros_like(steer))
        new_v.append(vel[k] + change[k] * _f32(BOIDS["global_scale"]))
    speed = torch.sqrt(sum(v * v for v in new_v))
    scale = torch.where(speed > 1, 1.0 / speed, torch.where(speed < 0.5, 0.5 / speed, torch.ones_like(speed)))
    for k in range(3):
        v = new_v[k] * scale
        if not wrap:
            v = v + (pos[k] < _f32(0.1)).double() * _f32(0.05) - (width - pos[k] < _f32(0.1)).double() * _f32(0.05)
        p = pos[k] + v * _f32(BOIDS["time_scale"])
        if wrap:
            p = torch.where(p < 0, p + width, p)
            p = torch.where(p > width, p - width, p)
        else:
            p = p.clamp(0.0, width)
        new_v[k] = v
        new_p.append(p)
    # from bin order back to the population's, then to the order of the agent sort
    out = {}
    final = _sort_order(pos32, edge, cells)
    for name, v in zip(F3, new_p + new_v):
        back = torch.empty_like(v)
        back[order] = v
        out[name] = back[final]
    return out


def _exact_payload(case, cols):
    edge, r = _payload_shape(case)
    dims, cells = case["dims"], int(math.ceil(np.float32(edge) / np.float32(r)))
    names = ("x", "y", "z")[:dims]
    pos32 = [cols[k] for k in names]
    cell, order, counts, start = _binned(pos32, r, cells)
    pos = [p.double()[order] for p in pos32]
    pay = [cols[f"p{k}"].double()[order] for k in range(4)]
    n = case["n"]
    for _ in range(case["steps"]):
        sums = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(4)]
        seen = torch.zeros(n, dtype=torch.float64, device="cuda")
        for pair in _neighbours(cells, dims, counts, start, False, cell, 3_000_000_000):
            if pair is None:
                return None
            a, m = pair
            inside = (sum((pos[k][m] - pos[k][a]) ** 2 for k in range(dims)) < r * r)
            a, m = a[inside], m[inside]
            seen[a] += 1.0
            for k in range(4):
                sums[k][a] += pay[k][m]
        pay = [torch.where(seen > 0, 0.5 * pay[k] + 0.5 * sums[k] / seen.clamp(min=1.0), pay[k]) for k in range(4)]
    out = {}
    final = _sort_order(pos32, edge, cells)
    for k in range(4):
        back = torch.empty_like(pay[k])
        back[order] = pay[k]
        out[f"p{k}"] = back[final]
    for k in names:
        out[k] = cols[k].double()[final]
    return out
