"""The workloads this library's performance is judged by, and their inputs.

A case is one call sequence of a user's program over seeded synthetic inputs:

  step   positions into a prepared handle, one reduction, the per-node results
         out, all in device memory (reset_node_data / IrregularStart /
         get_reduction_result of a simulation that lives on the GPU);
  host   the same through the IrregularRuntime class with plain (pageable) FP64
         host arrays, as the drivers this library replaces call it;
  init   a new edge list: handle, edges, nodes, set-up, one reduction, results
         (what a program pays each time its neighbour list changes);
  list   the half neighbour list of a set of positions;
  batch  many independent systems of different sizes reduced by one launch;
  md     a segment of a Lennard-Jones simulation: steps, energies, final state.

Systems are "gas" (a periodic or open box with every site of a sparse grid
displaced at random, nodes in random order: the moldyn-style random box, with
no pair close enough to overflow) or "fcc" (miniMD's lattice with thermal
displacements, nodes in lattice order).
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "ipdps15-pattern_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import irregular_gb300 as irr  # noqa: E402

MOLDYN, MINIMD, MINIMD_PBC = "moldyn", "minimd", "minimd_pbc"
_MAPS = {MOLDYN: irr.IRR_MAP_LJ_MOLDYN, MINIMD: irr.IRR_MAP_LJ_MINIMD, MINIMD_PBC: irr.IRR_MAP_LJ_MINIMD_PBC}
_FCC_DENSITY = 0.8442  # miniMD's reduced density


def _system_case(kind, place, n, density, cut, lst, law, node_bytes, out_bytes, **more):
    return dict({"kind": kind, "place": place, "n": n, "density": density, "cut": cut, "list": lst, "map": law,
                 "node_bytes": node_bytes, "out_bytes": out_bytes}, **more)


def listed():
    cases = {
        # the smallest system in earnest, 4 x 6^3 atoms in miniMD's lattice: launches and latency
        "step_864": _system_case("step", "fcc", 864, _FCC_DENSITY, 2.5, 2.8, MOLDYN, 24, 12),
        # 65,536 nodes with ~32 neighbours within 2.5: fits L2
        "step_65k": _system_case("step", "gas", 65536, 0.4889, 2.5, 2.5, MOLDYN, 12, 12),
        # miniMD's own problem: 500,000 atoms, open boundaries, list at cutoff + skin, FP64 records
        "step_minimd_500k": _system_case("step", "fcc", 500000, _FCC_DENSITY, 2.5, 2.8, MINIMD, 24, 24),
        # moldyn's own problem: 1,048,576 nodes with ~248 neighbours listed, cutoff 3.5
        "step_moldyn_1m": _system_case("step", "fcc", 1048576, 0.83134, 3.5, 4.145, MOLDYN, 16, 16),
        # the largest: 4,194,304 nodes with ~64 neighbours within 2.5
        "step_4m": _system_case("step", "gas", 4194304, 0.9778, 2.5, 2.5, MOLDYN, 12, 12),
        # the edge-parallel executor (no set-up to pay for), an odd size
        "plain_300k": _system_case("step", "gas", 300007, 0.9778, 2.5, 2.5, MOLDYN, 12, 12, plain=True),
        # the drop-in class on host arrays, results widened to the driver's double[3]
        "host_250k": _system_case("host", "gas", 250001, 0.83134, 2.5, 2.8, MOLDYN, 24, 24),
        # a new edge list, set up and reduced once
        "init_1m": _system_case("init", "gas", 1000003, 0.9778, 2.5, 2.5, MOLDYN, 12, 12),
        # a neighbour list
        "list_1m": _system_case("list", "gas", 1000003, 0.9778, 2.5, 2.8, MOLDYN, 12, 0),
        # 48 periodic systems, 2,000 to 120,000 nodes
        "batch_48": _system_case("batch", "gas", 2000, 0.83134, 2.5, 2.5, MINIMD_PBC, 12, 12, count=48,
                                 n_max=120000),
        # short simulations of miniMD's lattice: a small box and one that fills the GPU
        "md_32k": {"kind": "md", "cells": 20, "steps": 100},
        "md_864k": {"kind": "md", "cells": 60, "steps": 100},
    }
    return [dict(c, name=name) for name, c in cases.items()]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "plain", "host", "init", "list", "batch", "md"])
    if kind == "md":
        return {"kind": "md", "cells": _log_uniform(rng, 8, 56), "steps": rng.choice([20, 40, 60, 100])}
    density = rng.choice([0.4889, 0.83134, _FCC_DENSITY, 0.9778])
    neighbours = _log_uniform(rng, 20, 250 if kind == "step" else 100)
    lst = round((neighbours / density * 0.75 / math.pi) ** (1.0 / 3.0), 3)
    cut = lst if rng.random() < 0.4 else round(lst / 1.12, 3)
    top = {"step": 4000000, "plain": 400000, "host": 1000000, "init": 1500000, "list": 1500000, "batch": 20000}[kind]
    n = _log_uniform(rng, max(600, 6 * neighbours), max(1000, min(top, 64 * top // neighbours)))
    place = rng.choice(["gas", "fcc"])
    if kind == "batch":
        place, n = "gas", min(n, 20000)
    if place == "fcc":
        n = 4 * max(5, round((n / 4.0) ** (1.0 / 3.0))) ** 3
    law = rng.choice([MOLDYN, MOLDYN, MINIMD, MINIMD_PBC])
    node_bytes, out_bytes = rng.choice([(12, 12), (12, 12), (16, 16), (24, 12), (24, 24)])
    if kind == "plain":
        return _system_case("step", place, n, density, cut, lst, law, node_bytes, out_bytes, plain=True)
    if kind == "host":
        return _system_case("host", place, n, density, cut, lst, law, 24, rng.choice([12, 24]))
    if kind == "batch":
        count = rng.randint(6, 48)
        n_max = min(120000, n * rng.randint(2, 40))
        return _system_case("batch", place, n, density, cut, lst, rng.choice([MOLDYN, MINIMD_PBC]), 12, 12,
                            count=count, n_max=n_max)
    return _system_case(kind, place, n, density, cut, lst, law, node_bytes, out_bytes)


# ------------------------------------------------------------------ inputs

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFFFFFFFFFF)
    return g


def _positions(place, n, density, seed, spread=0.05):
    """(float64 (n, 3) positions on the GPU whose floats lie in [0, side), side);
    spread: the lattice's thermal displacement, in lattice constants."""
    g = _generator(seed)
    if place == "gas":
        side = float(np.float32((n / density) ** (1.0 / 3.0)))
        m = math.ceil((n / 0.8) ** (1.0 / 3.0))
        site = torch.randperm(m ** 3, generator=g, device="cuda")[:n]
        cell = torch.stack([site % m, site // m % m, site // (m * m)], dim=1).double()
        move = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * 0.6 - 0.3
        x = (cell + 0.5 + move) * (side / m)
    else:
        k = round((n / 4.0) ** (1.0 / 3.0))
        alat = (4.0 / density) ** (1.0 / 3.0)
        side = k * alat
        r = torch.arange(2 * k, device="cuda")
        z, y, x = torch.meshgrid(r, r, r, indexing="ij")
        keep = (x + y + z) % 2 == 0
        x = torch.stack([x[keep], y[keep], z[keep]], dim=1).double() * (0.5 * alat)
        x = x + torch.randn(x.shape, generator=g, device="cuda", dtype=torch.float64) * (spread * alat)
        x = torch.remainder(x, side)
    x[x.float() >= np.float32(side)] = 0.0
    return x.contiguous(), side


def _velocities(n, seed, temperature=1.44):
    v = torch.randn((n, 3), generator=_generator(seed + 1), device="cuda", dtype=torch.float64)
    v -= v.mean(dim=0)
    return v * math.sqrt(temperature * (3 * n - 3) / float((v * v).sum()))


def _records(x, node_bytes):
    if node_bytes == 24:
        return x
    if node_bytes == 12:
        return x.float().contiguous()
    return torch.cat([x.float(), torch.zeros_like(x[:, :1], dtype=torch.float32)], dim=1).contiguous()


def _params(case, side):
    if case["map"] == MOLDYN:
        return irr.moldyn_params(side, case["cut"])
    return irr.minimd_params(case["cut"] ** 2, None if case["map"] == MINIMD else side)


def _box(case, side):
    return 0.0 if case["map"] == MINIMD else side


def _list_cut2(case):
    return float(np.float32(case["list"] ** 2))


def _out(n, out_bytes):
    if out_bytes == 24:
        return torch.zeros((n, 3), device="cuda", dtype=torch.float64)
    return torch.zeros((n, out_bytes // 4), device="cuda", dtype=torch.float32)


def _handle(case, side, edges, nodes):
    """A handle on torch's current stream, ready for irr_init."""
    mode = irr.IRR_EXEC_PLAIN if case.get("plain") else irr.IRR_EXEC_PARTITIONED
    h = irr.Handle(irr.default_config(device=0, map_idx=_MAPS[case["map"]], exec=mode))
    h.set_stream(torch.cuda.current_stream().cuda_stream)
    h.set_params(_params(case, side))
    h.set_edges(edges)
    h.set_nodes(nodes)
    return h


def _batch_sizes(case):
    lo, hi, count = case["n"], case["n_max"], case["count"]
    return [int(round(lo * (hi / lo) ** (k / max(1, count - 1)))) for k in range(count)]


class _DeviceArray:
    """A library-owned edge list as torch sees it (kept alive by the tensor)."""

    def __init__(self, edges):
        self.edges = edges
        self.__cuda_array_interface__ = {"shape": (edges.count, 2), "typestr": "<i4", "data": (edges.ptr, False),
                                         "version": 3}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "md":
        n = 4 * case["cells"] ** 3
        x, side = _positions("fcc", n, _FCC_DENSITY, seed, 0.005)
        md = irr.MD(x.cpu().numpy(), _velocities(n, seed).cpu().numpy(), side)
        return {"case": case, "md": md}
    if kind == "batch":
        batch, handles, nodes = irr.Batch(0), [], []
        batch.set_stream(torch.cuda.current_stream().cuda_stream)
        for k, n in enumerate(_batch_sizes(case)):
            x, side = _positions(case["place"], n, case["density"], seed + 1000 * k)
            rec = _records(x, case["node_bytes"])
            h = _handle(case, side, irr.neighbor_build(x.float(), _box(case, side), _list_cut2(case)), rec)
            h.init()
            batch.add(h)
            handles.append(h)
            nodes.append(rec)
        batch.finalize()
        out = _out(sum(t.shape[0] for t in nodes), case["out_bytes"])
        parts = torch.split(out, [t.shape[0] for t in nodes])
        return {"case": case, "batch": batch, "handles": handles, "nodes": nodes, "out": out, "parts": parts}
    if kind == "list":
        # the seed numbers the nodes of one system: the pairs change, their count does not
        x, side = _positions(case["place"], case["n"], case["density"], case["n"])
        order = torch.randperm(case["n"], generator=_generator(seed), device="cuda")
        return {"case": case, "side": side, "pos": x[order].float().contiguous()}
    x, side = _positions(case["place"], case["n"], case["density"], seed)
    state = {"case": case, "side": side}
    edges = irr.neighbor_build(x.float(), _box(case, side), _list_cut2(case))
    if kind == "host":
        nodes = x.cpu().numpy()
        dt = np.float64 if case["out_bytes"] == 24 else np.float32
        rt = irr.IrregularRuntime(edges.count, case["n"], edges.to_host(), None, nodes, 0, 24, case["out_bytes"],
                                  parameter=_params(case, side), map_idx=_MAPS[case["map"]])
        rt.IrregularInit()
        return dict(state, rt=rt, nodes=nodes, out=np.zeros((case["n"], 3), dt))
    state["nodes"] = _records(x, case["node_bytes"])
    state["out"] = _out(case["n"], case["out_bytes"])
    if kind == "init":
        return dict(state, edges=edges)
    state["h"] = _handle(case, side, edges, state["nodes"])
    state["h"].init()
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        h = state["h"]
        h.set_nodes(state["nodes"])
        h.step()
        h.get_result_device(state["out"], case["out_bytes"])
        return state["out"]
    if kind == "batch":
        for h, rec in zip(state["handles"], state["nodes"]):
            h.set_nodes(rec)
        state["batch"].step()
        for h, part in zip(state["handles"], state["parts"]):
            h.get_result_device(part, case["out_bytes"])
        return state["out"]
    if kind == "host":
        rt = state["rt"]
        rt.reset_node_data(state["nodes"])
        rt.IrregularStart()
        return rt.get_reduction_result(state["out"])
    if kind == "init":
        h = _handle(case, state["side"], state["edges"], state["nodes"])
        h.init()
        h.step()
        h.get_result_device(state["out"], case["out_bytes"])
        h.close()
        return state["out"]
    if kind == "list":
        edges = irr.neighbor_build(state["pos"], _box(case, state["side"]), _list_cut2(case))
        if edges.count == 0:
            return torch.empty((0, 2), dtype=torch.int32, device="cuda")
        return torch.as_tensor(_DeviceArray(edges), device="cuda")
    md = state["md"]
    md.run(case["steps"])
    kinetic, potential, virial = md.energy()
    pos, vel = md.state()
    return {"kinetic": kinetic, "potential": potential, "virial": virial, "pos": pos, "vel": vel}


# -------------------------------------------------------- bytes, operations

def _pairs_expected(n, density, lst):
    return 0.5 * n * density * 4.0 / 3.0 * math.pi * lst ** 3


def work(case):
    """Each edge (8 bytes) and node record read once, each result written once;
    30 operations per pair of the law, 10 per listed pair of the list rule."""
    kind = case["kind"]
    if kind == "md":
        n, steps = 4 * case["cells"] ** 3, case["steps"]
        e = _pairs_expected(n, _FCC_DENSITY, 2.8)
        return {"bytes": steps * (8 * e + 96 * n) + 48 * n, "flops": steps * 30 * e}
    sizes = _batch_sizes(case) if kind == "batch" else [case["n"]]
    n = sum(sizes)
    e = _pairs_expected(n, case["density"], case["list"])
    return {"bytes": 8 * e + n * (case["node_bytes"] + case["out_bytes"]), "flops": (10 if kind == "list" else 30) * e}


# ------------------------------------------------------------- 64-bit values

def _half_pairs(p, box, cut2):
    """Pairs (i < j) of float positions with r2 <= cut2, by the list's rule in
    float: d wrapped once by +-box (0: open) when |d| > box / 2."""
    n = p.shape[0]
    cut = math.sqrt(cut2) * 1.001

    def hits(a, b):
        d = a - b
        if box:
            hb, bx = np.float32(0.5) * np.float32(box), float(np.float32(box))
            d = torch.where(d > float(hb), d - bx, torch.where(d < -float(hb), d + bx, d))
        d = d * d
        return (d[..., 0] + d[..., 1]) + d[..., 2] <= cut2

    lo = torch.zeros(3, device="cuda") if box else p.min(dim=0).values
    span = [box] * 3 if box else [float(s) for s in (p.max(dim=0).values - lo)]
    nc = [max(1, min(256, int(s / cut))) for s in span]
    if min(nc) < 3:
        i, j = torch.triu_indices(n, n, 1, device="cuda")
        keep = torch.cat([hits(p[a], p[b]) for a, b in zip(i.split(1 << 24), j.split(1 << 24))])
        return i[keep], j[keep]
    cells = torch.stack([((p[:, c] - lo[c]).double() / (span[c] / nc[c])).long().clamp(0, nc[c] - 1)
                         for c in range(3)], dim=1)
    key = (cells[:, 2] * nc[1] + cells[:, 1]) * nc[0] + cells[:, 0]
    order = torch.argsort(key)
    count = torch.bincount(key, minlength=nc[0] * nc[1] * nc[2])
    start = torch.cumsum(count, 0) - count
    slots = torch.arange(int(count.max()), device="cuda")
    q, at = p[order], cells[order]
    found = []
    forward = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1) if (z, y, x) >= (0, 0, 0)]
    for t0 in range(0, n, 1 << 17):
        t = torch.arange(t0, min(n, t0 + (1 << 17)), device="cuda")
        for off in forward:
            to = [at[t, c] + off[c] for c in range(3)]
            ok = torch.ones_like(t, dtype=torch.bool)
            for c in range(3):
                if box:
                    to[c] = to[c] % nc[c]
                else:
                    ok &= (to[c] >= 0) & (to[c] < nc[c])
                    to[c] = to[c].clamp(0, nc[c] - 1)
            k = (to[2] * nc[1] + to[1]) * nc[0] + to[0]
            u = start[k][:, None] + slots
            valid = ok[:, None] & (slots < count[k][:, None])
            if off == (0, 0, 0):
                valid &= u > t[:, None]
            u = u.clamp(max=n - 1)
            valid &= hits(q[t][:, None, :], q[u])
            row, slot = valid.nonzero(as_tuple=True)
            found.append(torch.stack([order[t[row]], order[u[row, slot]]]))
    i, j = torch.cat(found, dim=1)
    return torch.minimum(i, j), torch.maximum(i, j)


def _law(x, i, j, cut, side):
    """FP64 per-node sums of d (rd^-7 - rd^-4 / 2), the potential and the
    virial (force 48 x) over the pairs (i, j) inside the cutoff."""
    f = torch.zeros_like(x)
    potential = virial = 0.0
    for a, b in zip(i.split(1 << 24), j.split(1 << 24)):
        d = x[a] - x[b]
        if side:
            d = torch.where(d < -0.5 * side, d + side, torch.where(d > 0.5 * side, d - side, d))
        rd = (d * d).sum(dim=1)
        r = torch.where(rd < cut * cut, 1.0 / rd, torch.zeros_like(rd))
        r3 = r * r * r
        s = r3 * (r3 - 0.5) * r
        f.index_add_(0, a, d * s[:, None])
        f.index_add_(0, b, d * -s[:, None])
        potential += float((4.0 * r3 * (r3 - 1.0)).sum())
        virial += float((48.0 * s * rd).sum())
    return f, potential, virial


def _exact_md(case, seed):
    """Velocity Verlet with the list rebuilt every 20 steps at cutoff + skin."""
    n, dt = 4 * case["cells"] ** 3, 0.005
    x, side = _positions("fcc", n, _FCC_DENSITY, seed, 0.005)
    v = _velocities(n, seed)

    def pairs():
        p = x.float()
        return _half_pairs(torch.where(p >= np.float32(side), torch.zeros_like(p), p), side,
                           float(np.float32((2.5 + 0.3) ** 2)))

    i, j = pairs()
    f, potential, virial = _law(x, i, j, 2.5, side)
    for step in range(1, case["steps"] + 1):
        v = v + 0.5 * dt * 48.0 * f
        x = torch.remainder(x + dt * v, side)
        if step % 20 == 0:
            i, j = pairs()
        f, potential, virial = _law(x, i, j, 2.5, side)
        v = v + 0.5 * dt * 48.0 * f
    return {"kinetic": 0.5 * float((v * v).sum()), "potential": potential, "virial": virial, "pos": x, "vel": v}


def exact(case, seed):
    """Positions are used in float (so documented), the rest is FP64."""
    kind = case["kind"]
    if kind == "list":
        return None
    if kind == "md":
        return _exact_md(case, seed)
    if kind == "batch":
        systems = [(n, seed + 1000 * k) for k, n in enumerate(_batch_sizes(case))]
    else:
        systems = [(case["n"], seed)]
    parts = []
    for n, sd in systems:
        x, side = _positions(case["place"], n, case["density"], sd)
        p = x.float()
        i, j = _half_pairs(p, _box(case, side), _list_cut2(case))
        f = _law(p.double(), i, j, case["cut"], _box(case, side))[0]
        parts.append(torch.cat([f, torch.zeros_like(f[:, :1])], dim=1) if case["out_bytes"] == 16 else f)
    return torch.cat(parts)
