"""The workloads this library is timed on, with their inputs.

Each case is one call (or, for the server, one burst of calls) of a public
entry point on inputs that are made from a seed.  The listed cases are the
structures of the benchmark (``neighborlist_rs.workloads``) and the sizes
around them: the unit cell a relaxation asks for at every step, the isolated
molecule, the 10,008-atom liquid at a short and a long cutoff, a million
atoms, the edge vectors a graph network is fed with, a molecular-dynamics
step, the numpy entry points, thousands of small systems in one call, and a
burst of served requests.  ``draw`` gives further cases of the same kinds over
the same ranges of atoms, cutoffs, cells and options.

    listed()             the cases
    draw(rng)            one more case
    prepare(case, seed)  the inputs and handles a program has before the call
    run(state)           one pass, and what it returns
    work(case)           the bytes and operations a pass cannot do without
    exact(case, seed)    the floating outputs in plain numpy, 64 bits
"""

import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "neighborlist-rs_b200"))

import neighborlist_rs as nl  # noqa: E402
from neighborlist_rs import workloads  # noqa: E402
from neighborlist_rs.serving import Server  # noqa: E402
from neighborlist_rs.verlet import VerletList  # noqa: E402

DENSITY = 0.1  # atoms per cubic Angstrom, as in the benchmark
LIQUID_BOX = 46.4  # holds 1112 clusters of 9 atoms
LARGEST = 1_000_000 * 6.0 ** 3  # atoms x cutoff^3 of the largest listed case


def listed():
    return [
        # A relaxation of a small periodic cell with the positions on the
        # GPU: the cell is narrower than two cutoffs, latency is everything.
        {"name": "cell_60", "kind": "device", "shape": "triclinic", "n": 60, "rc": 5.0},
        # One isolated molecule or cluster (no cell), on the GPU.
        {"name": "isolated_1000", "kind": "device", "shape": "isolated", "n": 1000, "rc": 6.0},
        # The benchmark's liquid at its short and its long cutoff, on the GPU.
        {"name": "liquid_10008_rc6", "kind": "device", "shape": "liquid", "n": 10008, "rc": 6.0},
        {"name": "liquid_10008_rc14", "kind": "device", "shape": "liquid", "n": 10008, "rc": 14.0},
        # The largest structure the server and the tests take, on the GPU.
        {"name": "bulk_1000000", "kind": "device", "shape": "ortho", "n": 1_000_000, "rc": 6.0},
        # What a graph network is fed with: directed edges with their vectors
        # and lengths, in a skewed cell.
        {"name": "edges_20001", "kind": "edges", "shape": "triclinic", "n": 20001, "rc": 5.0,
         "directed": True, "vectors": True, "distances": True},
        # One molecular-dynamics step: the skin list filtered at the cutoff.
        {"name": "md_10008", "kind": "verlet", "shape": "liquid", "n": 10008, "rc": 6.0,
         "skin": 1.0},
        # The drop-in call: numpy in, numpy out.
        {"name": "host_liquid_10008", "kind": "host", "shape": "liquid", "n": 10008, "rc": 6.0},
        # The benchmark's multi-cutoff structure: three lists from one call.
        {"name": "host_multi_20000", "kind": "multi", "shape": "triclinic", "n": 20000,
         "rc": 12.0, "rc1": 5.0, "rc2": 6.0, "disjoint": False},
        # A data set of uneven small systems in one call, half of them
        # isolated, half in skewed cells.
        {"name": "batch_4096", "kind": "batch", "systems": 4096, "lo": 8, "hi": 256, "rc": 5.0},
        # A training batch with two disjoint shells per system.
        {"name": "batch_shells_333", "kind": "batch_multi", "systems": 333, "lo": 8, "hi": 256,
         "rc": 5.0, "rc1": 3.0, "disjoint": True},
        # A burst of requests of mixed sizes to the server, results on the
        # GPU (sizes, cells and cutoffs of the served distribution).
        {"name": "served_30", "kind": "served", "requests": 30, "lo": 16, "hi": 100_000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _atoms(rng, lo, hi, rc):
    return _log_int(rng, lo, max(lo, min(hi, int(LARGEST / rc ** 3))))


def draw(rng):
    kind = rng.choice(["device"] * 5 + ["edges", "verlet", "host", "multi", "batch",
                                        "batch_multi", "served"])
    shape = rng.choice(["ortho", "triclinic", "isolated", "liquid"])
    if kind == "device":
        rc = rng.choice([5.0, 6.0, 8.0, 14.0])
        return {"kind": kind, "shape": shape, "n": _atoms(rng, 16, 1_000_000, rc), "rc": rc}
    if kind == "edges":
        return {"kind": kind, "shape": shape, "n": _atoms(rng, 16, 60_000, 5.0),
                "rc": rng.choice([5.0, 6.0]), "directed": rng.random() < 0.7,
                "vectors": True, "distances": rng.random() < 0.7}
    if kind == "verlet":
        rc = rng.choice([5.0, 6.0, 8.0, 14.0])
        return {"kind": kind, "shape": rng.choice(["ortho", "triclinic", "liquid"]),
                "n": _atoms(rng, 200, 100_000, 1.7 * rc), "rc": rc,
                "skin": round(rng.uniform(0.8, 2.0), 2)}
    if kind == "host":
        rc = rng.choice([5.0, 6.0, 8.0, 14.0])
        return {"kind": kind, "shape": shape, "n": min(_atoms(rng, 16, 200_000, rc),
                                                       int(2e7 / rc ** 3)), "rc": rc}
    if kind == "multi":
        return {"kind": kind, "shape": shape, "n": _log_int(rng, 16, 20_000),
                "rc": rng.choice([8.0, 12.0]), "rc1": 5.0, "rc2": 6.0,
                "disjoint": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "systems": _log_int(rng, 8, 4096), "lo": 8,
                "hi": rng.choice([32, 100, 256]), "rc": rng.choice([4.0, 5.0, 6.0])}
    if kind == "batch_multi":
        return {"kind": kind, "systems": _log_int(rng, 8, 1024), "lo": 8,
                "hi": rng.choice([32, 100, 256]), "rc": rng.choice([5.0, 6.0]), "rc1": 3.0,
                "disjoint": rng.random() < 0.5}
    return {"kind": kind, "requests": rng.randint(4, 30), "lo": 16,
            "hi": rng.choice([2048, 20_000, 100_000])}


def _moved(pos, rows, rng, block=1):
    """The same structure as another program has it: its atoms (or clusters of
    `block` atoms) in another order and all of it moved by one vector, so that
    every position, bin and image differs and only the number of edges stays."""
    whole = len(pos) // block * block
    mixed = pos[:whole].reshape(-1, block, 3)[rng.permutation(whole // block)].reshape(-1, 3)
    by = rng.random(3) @ (np.eye(3) * 10.0 if rows is None else rows)
    return np.concatenate([mixed, pos[whole:]]) + by


def _base(shape, n):
    """(positions (N, 3), cell rows or None) of n atoms at DENSITY."""
    rng = np.random.default_rng(n)
    if shape == "isolated":
        return rng.random((n, 3)) * (n / DENSITY) ** (1.0 / 3.0), None
    if shape == "liquid":
        clusters = -(-n // 9)
        box = LIQUID_BOX * (clusters / 1112.0) ** (1.0 / 3.0)
        kept = min(clusters, 1112)  # distinct clusters; more reuse their shapes
        pos, _ = workloads.cluster_liquid(n_clusters=kept, box=box, seed=n)
        if clusters > kept:
            shapes = pos.reshape(kept, 9, 3)
            shapes = shapes - shapes.mean(axis=1, keepdims=True)
            pos = (shapes[rng.integers(0, kept, clusters)]
                   + rng.random((clusters, 1, 3)) * box).reshape(-1, 3)
        return np.ascontiguousarray(pos[:n]), np.diag([box, box, box])
    rows = workloads.density_cell(n, DENSITY, rng, (75.0, 105.0), ortho=shape == "ortho")
    return rng.random((n, 3)) @ rows, rows


def _structure(case, seed):
    """The positions and cell rows of a single-system case, and for a
    molecular-dynamics step also the positions its list was built at."""
    pos, rows = _base(case["shape"], case["n"])
    if case["kind"] == "verlet":
        # moved by up to 0.35 skin from the list's positions: the step filters
        rng = np.random.default_rng(7)
        move = rng.normal(size=pos.shape)
        move *= (rng.random((len(pos), 1)) ** (1.0 / 3.0) * 0.35 * case["skin"]
                 / np.linalg.norm(move, axis=1, keepdims=True))
        pos = np.concatenate([pos, pos + move], axis=1)
        mixed = np.random.default_rng(seed).permutation(len(pos))
        return pos[mixed, 3:], rows, pos[mixed, :3]
    block = 9 if case["shape"] == "liquid" else 1
    return _moved(pos, rows, np.random.default_rng(seed), block), rows


def _cell(rows):
    return None if rows is None else nl.PyCell(rows.T.tolist())


def _cutoffs(case):
    return [case[k] for k in ("rc1", "rc2", "rc") if k in case]


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("batch", "batch_multi"):
        systems = workloads.uneven_batch(case["systems"], (case["lo"], case["hi"]), DENSITY)
        rng = np.random.default_rng(seed)
        systems = [workloads.System(_moved(s.positions, s.cell_rows, rng), s.cell_rows, s.cutoff)
                   for s in (systems[k] for k in rng.permutation(len(systems)))]
        pos, batch, cells = workloads.concat_batch(systems)
        return {"case": case, "pos": pos, "batch": batch, "cells": cells}
    if kind == "served":
        reqs = workloads.request_stream(case["requests"], 5, (case["lo"], case["hi"]), DENSITY)
        rng = np.random.default_rng(seed)
        return {"case": case, "server": Server(hbm_budget_bytes=8 << 30, workers=4),
                "requests": [(_cell(s.cell_rows), _moved(s.positions, s.cell_rows, rng), s.cutoff)
                             for s in reqs]}
    pos, rows, *reference = _structure(case, seed)
    state = {"case": case, "cell": _cell(rows), "pos": pos}
    if kind in ("device", "edges", "verlet"):
        state["pos"] = torch.from_numpy(pos).cuda()
    if kind == "verlet":
        state["list"] = VerletList(case["rc"], case["skin"])
        state["list"].update(state["cell"], torch.from_numpy(reference[0]).cuda())
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "device":
        return nl.build_neighborlists_torch(state["cell"], state["pos"], case["rc"])
    if kind == "edges":
        return nl.build_neighborlists_torch(
            state["cell"], state["pos"], case["rc"], directed=case["directed"],
            vectors=case["vectors"], distances=case["distances"])
    if kind == "verlet":
        return state["list"].update(state["cell"], state["pos"])
    if kind == "host":
        return nl.build_neighborlists(state["cell"], state["pos"], case["rc"])
    if kind == "multi":
        return nl.build_neighborlists_multi(state["cell"], state["pos"], _cutoffs(case),
                                            disjoint=case["disjoint"])
    if kind == "batch":
        return nl.build_neighborlists_batch(state["pos"], state["batch"], state["cells"],
                                            case["rc"])
    if kind == "batch_multi":
        return nl.build_neighborlists_batch_multi(state["pos"], state["batch"], state["cells"],
                                                  _cutoffs(case), disjoint=case["disjoint"])
    server = state["server"]
    tickets = [server.submit(c, p, rc, device_result=True) for c, p, rc in state["requests"]]
    out = []
    for t in tickets:
        result = server.wait(t)
        out.append(result.to_torch())
        result.release()
    return out


def _pairs(n, rc, isolated):
    """Expected edges of n atoms at DENSITY (a cube without a cell: the
    distribution of distances in a cube)."""
    if not isolated:
        return n * DENSITY * 4.0 / 3.0 * math.pi * rc ** 3 / 2.0
    x = min(1.0, rc / (n / DENSITY) ** (1.0 / 3.0))
    inside = 4.0 / 3.0 * math.pi * x ** 3 - 1.5 * math.pi * x ** 4 + 1.6 * x ** 5 - x ** 6 / 6.0
    return n * (n - 1) / 2.0 * inside


def work(case):
    """Positions (24 bytes an atom) and cells read once, every edge (two int64
    and three int32) written once, vectors and lengths 24 and 8 bytes an
    edge; 8 operations for the distance of each edge."""
    kind = case["kind"]
    atoms, cells, edges, extra = case.get("n", 0), 1.0, 0.0, 0.0
    if kind in ("batch", "batch_multi"):
        sizes = range(case["lo"], case["hi"] + 1)
        mean = sum(sizes) / len(sizes)
        atoms, cells = case["systems"] * mean, case["systems"]
        for rc in [max(_cutoffs(case))] if case.get("disjoint") else _cutoffs(case):
            edges += cells * sum(_pairs(n, rc, False) + _pairs(n, rc, True)
                                 for n in sizes) / (2.0 * len(sizes))
    elif kind == "served":
        lo, hi = math.log(case["lo"]), math.log(case["hi"])
        mean = (case["hi"] - case["lo"]) / (hi - lo)
        atoms, cells = case["requests"] * mean, case["requests"]
        edges = sum(_pairs(atoms, rc, False) for rc in (5.0, 6.0, 8.0)) / 3.0
    elif kind == "verlet":
        # the stored list at rc + skin is read, the kept edges are written
        edges = _pairs(atoms, case["rc"], False)
        extra = 28.0 * _pairs(atoms, case["rc"] + case["skin"], False)
    else:
        isolated = case["shape"] == "isolated"
        for rc in [case["rc"]] if case.get("disjoint") else _cutoffs(case):
            edges += _pairs(atoms, rc, isolated)
        if kind == "edges":
            edges *= 2.0 if case["directed"] else 1.0
            extra = edges * (24.0 * case["vectors"] + 8.0 * case["distances"])
    return {"bytes": 24.0 * atoms + 72.0 * cells + 28.0 * edges + extra, "flops": 8.0 * edges}


def _spread(v):
    """Every bit of v (21 bits) moved to three times its place."""
    out = np.zeros_like(v)
    for b in range(21):
        out |= ((v >> b) & 1) << (3 * b)
    return out


def _half_list(pos, h, rc):
    """The half list of a cell-list build (h: columns are the lattice
    vectors) in its canonical order: atoms by bin and position along the
    Z-order curve, stencil cells x outer to z inner, candidates in the atoms'
    order.  Returns (i, j, shift)."""
    hinv = np.linalg.inv(h)
    width = 1.0 / np.linalg.norm(hinv, axis=1)
    nb = np.maximum(1, np.floor(width / rc)).astype(np.int64)
    ns = np.ceil(rc * nb / width).astype(np.int64)
    frac = pos @ hinv.T
    low = np.floor(frac)
    u = frac - low
    wrapped = pos - low @ h.T
    s = -low.astype(np.int64)
    bins = np.minimum((u * nb).astype(np.int64), nb - 1)
    fine = (np.clip(u, 0.0, 0.999999) * 2097152.0).astype(np.int64)
    code = [_spread(v[:, 0]) | _spread(v[:, 1]) << 1 | _spread(v[:, 2]) << 2 for v in (bins, fine)]
    order = np.lexsort((np.arange(len(pos)), code[1], code[0]))
    w, b = wrapped[order], bins[order]
    linear = b[:, 0] + nb[0] * (b[:, 1] + nb[1] * b[:, 2])
    start = np.full(int(nb.prod()), 0)
    count = np.bincount(linear, minlength=int(nb.prod()))
    first = np.unique(linear, return_index=True)
    start[first[0]] = first[1]
    found = []
    for ix in range(-ns[0], ns[0] + 1):
        for iy in range(-ns[1], ns[1] + 1):
            for iz in range(-ns[2], ns[2] + 1):
                at = b + np.array([ix, iy, iz])
                image = np.floor_divide(at, nb)
                at = at - image * nb
                target = at[:, 0] + nb[0] * (at[:, 1] + nb[1] * at[:, 2])
                k = count[target]
                i = np.repeat(np.arange(len(pos)), k)
                j = np.arange(len(i)) - np.repeat(np.cumsum(k) - k - start[target], k)
                d = (w[j] - w[i]) + (image @ h.T)[i]
                near = (d * d).sum(axis=1) < rc * rc
                i, j = i[near], j[near]
                oi, oj = order[i], order[j]
                half = (oi < oj) | ((oi == oj) & image[i].any(axis=1))
                found.append((i[half], oi[half], oj[half],
                              s[oj[half]] - s[oi[half]] + image[i[half]]))
    at, i, j, shift = (np.concatenate(v) for v in zip(*found))
    by_atom = np.argsort(at, kind="stable")
    return i[by_atom], j[by_atom], shift[by_atom]


def exact(case, seed):
    """Vectors and lengths of an edge list (None for the list itself and for
    the other cases, which return whole numbers)."""
    if case["kind"] != "edges" or case["n"] > 60_000:
        return None
    pos, rows = _structure(case, seed)
    if rows is None:
        # no cell: a box one cutoff and 1 Angstrom wider on every side orders
        # the atoms; below 1000 atoms the pairs come in index order
        h = np.diag(pos.max(axis=0) - pos.min(axis=0) + 2.0 * (case["rc"] + 1.0))
    else:
        h = rows.T
    width = 1.0 / np.linalg.norm(np.linalg.inv(h), axis=1)
    if len(pos) < 1000 and 2.0 * case["rc"] < width.min():
        i, j = np.triu_indices(len(pos), 1)
        d = pos[j] - pos[i]
        shift = np.zeros((len(i), 3))
        if rows is not None:
            shift = -np.rint(d @ np.linalg.inv(h).T)
        d = d + shift @ h.T
        near = (d * d).sum(axis=1) < case["rc"] ** 2
        d = d[near]
    else:
        i, j, shift = _half_list(pos, h, case["rc"])
        d = (pos[j] - pos[i]) + (0.0 if rows is None else shift @ h.T)
    if case["directed"]:
        d = np.concatenate([d, -d])
    out = {"edge_index": None, "shift": None, "vectors": d}
    if case["distances"]:
        out["distances"] = np.sqrt((d * d).sum(axis=1))
    return out
