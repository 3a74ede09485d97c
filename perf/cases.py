"""The performance cases: what a program that uses vite_b200 has it do, over the real range.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare` makes what the
program holds before the call, `run` is one pass through the public entry points, `work` the bytes
and operations a pass cannot do without, and `exact` the floating-point outputs in plain numpy.

Families of graphs, as in the benchmark and the tests: `rgg` (Vite's in-memory random geometric
graph: radius r(n), average degree 7 to 12, plus 1 % random edges), `er` (Erdos-Renyi) and `ba`
(Barabasi-Albert, with hubs). Weights: `dist` (the generator's own: distances, and U(0,1) on the
random edges), `unit` (SET_EDGE_WEIGHTS_TO_ONE) or `u01` (U(0,1) per pair). Graphs below
HOST_VERTICES are drawn here on the host and uploaded, as small requests arrive; larger ones come
from the device generators.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import vite_b200

HOST_VERTICES = 40_000
EXACT_ENTRIES = 700_000  # the plain numpy phase loop stays within seconds up to here
THRESHOLD = 1e-6
LEVELS = 32  # more levels than a run has

_shared = {}


def _ctx() -> vite_b200.Context:
    """One context for the process, as a program that runs many graphs keeps it."""
    if "ctx" not in _shared:
        _shared["ctx"] = vite_b200.Context(0)
    return _shared["ctx"]


def listed() -> list:
    return [
        # the smallest request: its time is launches and read-backs
        {"name": "run_rgg_1k", "kind": "run", "family": "rgg", "n": 1201, "deg": 0, "weights": "dist"},
        # an ordinary small request without locality, unit weights (many ties)
        {"name": "run_er_20k", "kind": "run", "family": "er", "n": 20_011, "deg": 16, "weights": "unit"},
        # a middling geometric graph, just large enough for the locality layout
        {"name": "run_rgg_300k", "kind": "run", "family": "rgg", "n": 300_007, "deg": 0, "weights": "dist"},
        # the benchmark's headline: the largest geometric graph, device-resident
        {"name": "run_rgg_16m", "kind": "run", "family": "rgg", "n": 1 << 24, "deg": 0, "weights": "dist"},
        # a large preferential-attachment graph with real weights (hubs, coarse dense levels)
        {"name": "run_ba_2m_u01", "kind": "run", "family": "ba", "n": 2_266_207, "deg": 8, "weights": "u01"},
        # coloring and early termination, the benchmark's second configuration (-c 8 -t 2 -a 0.25)
        {"name": "run_ba_4m_c8_t2", "kind": "run", "family": "ba", "n": 1 << 22, "deg": 8,
         "weights": "unit", "coloring": True, "max_colors": 8, "et_type": 2, "et_delta": 0.25},
        # threshold cycling with early termination by frozen share (-i -t 3)
        {"name": "run_rgg_1m_i_t3", "kind": "run", "family": "rgg", "n": 1_000_003, "deg": 0,
         "weights": "unit", "threshold_scaling": True, "et_type": 3},
        # many mixed small graphs as one batch (the batched workload's size range and mix)
        {"name": "batch_48", "kind": "batch", "n": 48, "low": 1000, "high": 256_000, "mix": 4242},
        # the operator calls a host program makes level by level: hand-off of its CSR, one phase,
        # the communities back, the coarse graph built, its degrees and its own phase
        {"name": "level_er_200k", "kind": "level", "family": "er", "n": 200_003, "deg": 16, "weights": "u01"},
        # weighted degrees without allocation, rows from empty to hubs, real weights
        {"name": "degree_2m", "kind": "degree", "n": 2_000_003, "deg": 8, "weights": "u01"},
        # the multi-hash coloring alone, 70 % coverage
        {"name": "color_rgg_2m", "kind": "color", "family": "rgg", "n": 2_000_003, "deg": 0,
         "weights": "unit", "n_hash": 4},
        # ground-truth comparison of two label vectors in host memory
        {"name": "compare_1m", "kind": "compare", "n": 1_000_003, "mean": 64},
    ]


def _log_int(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["run", "run", "run", "run", "run", "batch", "level", "degree", "color", "compare"])
    if kind == "batch":
        low = _log_int(rng, 1000, 8000)
        return {"kind": kind, "n": rng.randint(3, 56), "low": low,
                "high": _log_int(rng, 2 * low, 256_000), "mix": rng.randint(1, 10**6)}
    if kind == "compare":
        return {"kind": kind, "n": _log_int(rng, 1000, 4_000_000), "mean": _log_int(rng, 4, 4000)}
    family = rng.choice(["rgg", "er", "ba"])
    if kind == "degree":
        return {"kind": kind, "n": _log_int(rng, 1000, 8_000_000), "deg": rng.randint(2, 16),
                "weights": rng.choice(["unit", "u01"])}
    weights = rng.choice(["unit", "u01", "dist"] if family == "rgg" else ["unit", "u01"])
    deg = 0 if family == "rgg" else rng.randint(4, 20) if family == "er" else rng.randint(2, 9)
    if kind == "color":
        return {"kind": kind, "family": family, "n": _log_int(rng, 1000, 4_000_000), "deg": deg,
                "weights": "unit", "n_hash": rng.randint(1, 8)}
    if kind == "level":
        return {"kind": kind, "family": family, "n": _log_int(rng, 1000, 500_000), "deg": deg,
                "weights": weights}
    case = {"kind": kind, "family": family, "deg": deg, "weights": weights,
            "n": _log_int(rng, 1000, 8_000_000 if family == "rgg" else 1_500_000)}
    option = rng.choice(["plain", "plain", "plain", "color", "order", "et", "cycle"])
    if option == "color":
        case |= {"coloring": True, "max_colors": 8}
    elif option == "order":
        case |= {"vertex_order": True, "max_colors": 8}
    elif option == "et":
        case |= {"et_type": rng.randint(1, 4), "et_delta": rng.choice([0.25, 0.5, 0.75])}
    elif option == "cycle":
        case |= {"threshold_scaling": True}
    return case


# ------------------------------------------------------------------------------------
# inputs

def _radius(n: int) -> float:
    return (math.sqrt(math.log(n) / (3.14159 * n)) + math.sqrt(2.0736 / n)) / 2.0


def _csr(n: int, u, v, w):
    """CSR with both directions of the undirected pairs (u < v, unique), rows sorted by tail."""
    src, dst, ww = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.argsort(src * n + dst, kind="stable")
    rowptr = np.zeros(n + 1, np.int64)
    rowptr[1:] = np.cumsum(np.bincount(src, minlength=n))
    return rowptr, dst[order], ww[order]


def _unique_pairs(n: int, a, b):
    lo, hi = np.minimum(a, b), np.maximum(a, b)
    keys = np.unique((lo * n + hi)[lo != hi])
    return keys // n, keys % n


def _host_graph(case: dict, seed: int):
    """(rowptr, tail, weight) of a small graph, from the seed alone."""
    rng = np.random.default_rng([seed, case["n"], case["deg"]])
    n = case["n"]
    dist = None
    if case["family"] == "rgg":
        r = _radius(n)
        xy = rng.random((n, 2))
        k = max(1, int(1.0 / r))
        cell = (xy * k).astype(np.int64).clip(0, k - 1)
        cid = cell[:, 0] * k + cell[:, 1]
        order = np.argsort(cid, kind="stable")
        start = np.searchsorted(cid[order], np.arange(k * k + 1))
        a, b = [], []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                x, y = cell[:, 0] + dx, cell[:, 1] + dy
                ok = (x >= 0) & (x < k) & (y >= 0) & (y < k)
                c = np.where(ok, x * k + y, 0)
                lo, cnt = start[c], np.where(ok, start[c + 1] - start[c], 0)
                for j in range(int(cnt.max())):
                    i = np.flatnonzero(cnt > j)
                    o = order[lo[i] + j]
                    near = (i < o) & (np.hypot(*(xy[i] - xy[o]).T) <= r)
                    a.append(i[near])
                    b.append(o[near])
        extra = max(1, sum(map(len, a)) // 100)
        a.append(rng.integers(0, n, extra))
        b.append(rng.integers(0, n, extra))
        u, v = _unique_pairs(n, np.concatenate(a), np.concatenate(b))
        dist = np.hypot(*(xy[u] - xy[v]).T)
        far = dist > r
        dist[far] = rng.random(int(far.sum()))
    elif case["family"] == "er":
        m = n * case["deg"] // 2
        u, v = _unique_pairs(n, rng.integers(0, n, m), rng.integers(0, n, m))
    else:  # endpoint slots of preferential attachment: a slot copies an earlier one
        m = case["deg"]
        e = n * m
        pick = (rng.random(e) * (2 * np.arange(e) + 1)).astype(np.int64)
        while True:  # odd slots hold copies: follow them to a vertex's own slot
            odd = (pick & 1) == 1
            if not odd.any():
                break
            pick[odd] = pick[pick[odd] // 2]
        u, v = _unique_pairs(n, np.arange(e) // m, (pick // 2) // m)
    if case["weights"] == "unit":
        w = np.ones(len(u))
    elif case["weights"] == "u01":
        w = rng.random(len(u))
    else:
        w = dist
    return _csr(n, u, v, w)


def _device_graph(ctx, case: dict, seed: int) -> vite_b200.Graph:
    if case["n"] < HOST_VERTICES:
        return ctx.upload(*_host_graph(case, seed))
    n = case["n"]
    if case["family"] == "rgg":
        g = ctx.generate_rgg(n, 1.0, 1 + seed)
    elif case["family"] == "er":
        g = ctx.generate_er(n, float(case["deg"]), 1 + seed)
    else:
        g = ctx.generate_ba(n, case["deg"], 1 + seed)
    if case["weights"] == "unit":
        ctx.reweight(g, 1)
    elif case["weights"] == "u01":
        ctx.reweight(g, 2, 7919 + seed)
    return g


def _pinned(a: np.ndarray) -> np.ndarray:
    """A page-locked copy, the host memory a program hands over and receives in."""
    t = torch.empty(max(a.nbytes, 1), dtype=torch.uint8, pin_memory=True)
    out = t.numpy()[:a.nbytes].view(a.dtype).reshape(a.shape)
    out[...] = a
    return out


def _batch_case(case: dict, i: int) -> dict:
    """Graph i of a batch: n log-uniform in [low, high], half rgg and half er, unit or u01."""
    r = np.random.default_rng([case["mix"], i])
    n = int(math.exp(r.uniform(math.log(case["low"]), math.log(case["high"]))))
    return {"family": ("rgg", "er")[i % 2], "n": n, "deg": 16 * (i % 2),
            "weights": ("unit", "u01")[int(r.integers(2))]}


def _degree_input(case: dict, seed: int):
    """A CSR's offsets and weights with preferential-attachment row lengths (some rows empty)."""
    rng = np.random.default_rng([seed, case["n"], case["deg"], 3])
    n, m = case["n"], case["deg"]
    d = np.minimum(m / np.sqrt(1.0 - rng.random(n)), 16.0 * math.sqrt(n)).astype(np.int64)
    d[rng.random(n) < 0.01] = 0
    rowptr = np.zeros(n + 1, np.int64)
    rowptr[1:] = np.cumsum(d)
    ne = int(rowptr[-1])
    return rowptr, np.ones(ne) if case["weights"] == "unit" else rng.random(ne)


def _compare_input(case: dict, seed: int):
    rng = np.random.default_rng([seed, case["n"], case["mean"], 5])
    n = case["n"]
    truth = np.arange(n, dtype=np.int64) // case["mean"]
    found = truth // 2
    move = rng.random(n) < 0.1
    found[move] = rng.integers(0, found.max() + 1, int(move.sum()))
    return truth, found


OPTIONS = ("coloring", "vertex_order", "max_colors", "et_type", "et_delta", "threshold_scaling")


def prepare(case: dict, seed: int):
    ctx = _ctx()
    kind = case["kind"]
    s = {"case": case, "ctx": ctx}
    if kind == "run":
        s["graph"] = _device_graph(ctx, case, seed)
        s["comm"] = _pinned(np.zeros(case["n"], np.int64))
        s["options"] = {k: case[k] for k in OPTIONS if k in case}
    elif kind == "batch":
        s["graphs"] = [_device_graph(ctx, _batch_case(case, i), 1000 * seed + i) for i in range(case["n"])]
    elif kind == "level":
        g = None
        if case["n"] < HOST_VERTICES:
            rowptr, tail, weight = _host_graph(case, seed)
        else:
            g = _device_graph(ctx, case, seed)
            rowptr, tail, weight = g.download()
            g.free()
        edges = np.empty(len(tail), vite_b200.EDGE_DTYPE)
        edges["tail"], edges["weight"] = tail, weight
        s["rowptr"], s["edges"] = _pinned(rowptr), _pinned(edges)
    elif kind == "degree":
        rowptr, weight = _degree_input(case, seed)
        s["rowptr"], s["weight"] = torch.from_numpy(rowptr).cuda(), torch.from_numpy(weight).cuda()
        s["vdeg"] = torch.empty(case["n"], dtype=torch.float64, device="cuda")
    elif kind == "color":
        s["graph"] = _device_graph(ctx, case, seed)
    else:
        s["truth"], s["found"] = _compare_input(case, seed)
    return s


# ------------------------------------------------------------------------------------
# one pass

def _padded(values, n: int, dtype) -> np.ndarray:
    """`values` and zeros: the number of levels and of communities differs from input to input."""
    out = np.zeros(n, dtype)
    out[:len(values)] = values
    return out


def _level_arrays(runs: list) -> dict:
    """What the program keeps of each run's levels, LEVELS places per run."""
    names = {"nv": np.int64, "ne": np.int64, "iters": np.int64, "num_colors": np.int64,
             "modularity": np.float64}
    return {k: np.concatenate([_padded([x[k] for x in r.stats], LEVELS, t) for r in runs])
            for k, t in names.items()}


def run(s):
    ctx, kind = s["ctx"], s["case"]["kind"]
    if kind == "run":
        r = ctx.run(s["graph"], threshold=THRESHOLD, comm_out=s["comm"], **s["options"])
        return {**_level_arrays([r]), "comm": r.comm}
    if kind == "batch":
        rs = ctx.run_batch(s["graphs"], threshold=THRESHOLD, want_comm=True)
        return {**_level_arrays(rs), "comm": [r.comm for r in rs]}
    if kind == "level":
        g = ctx.upload_edges(s["rowptr"], s["edges"])
        comm, modularity, iters = ctx.louvain_phase(g, threshold=THRESHOLD)
        ctx.rebuild(g)
        vdeg, constant = ctx.vertex_degree(g)
        comm2, modularity2, iters2 = ctx.louvain_phase(g, threshold=THRESHOLD)
        g.free()
        n = s["case"]["n"]
        return {"comm": comm, "modularity": modularity, "iters": iters, "constant": constant,
                "vdeg": _padded(vdeg, n, np.float64), "comm2": _padded(comm2, n, np.int64),
                "modularity2": modularity2, "iters2": iters2}
    if kind == "degree":
        c = vite_b200.vertex_degree_noalloc(
            s["case"]["n"], s["rowptr"].data_ptr(), s["weight"].data_ptr(), s["vdeg"].data_ptr(),
            stream=torch.cuda.current_stream().cuda_stream)
        return {"vdeg": s["vdeg"], "constant": c}
    if kind == "color":
        colors, count = ctx.color(s["graph"], s["case"]["n_hash"])
        return {"colors": colors, "count": count}
    return ctx.compare_communities(s["truth"], s["found"])


# ------------------------------------------------------------------------------------
# what a pass cannot do without

def _entries(case: dict) -> float:
    n = case["n"]
    if case["family"] == "rgg":
        return 1.01 * n * n * 3.14159 * _radius(n) ** 2
    return float(n * case["deg"]) if case["family"] == "er" else 2.0 * n * case["deg"]


def work(case: dict) -> dict:
    """A graph read once (rowptr 8 B; tail 4 B and weight 8 B per entry on the device, 16 B per
    entry from the host) and the results written once; one addition per entry."""
    n, kind = case["n"], case["kind"]
    if kind == "run":
        e = _entries(case)
        return {"bytes": 16.0 * n + 12.0 * e, "flops": e}
    if kind == "batch":
        sub = [_batch_case(case, i) for i in range(n)]
        e, v = sum(map(_entries, sub)), sum(c["n"] for c in sub)
        return {"bytes": 16.0 * v + 12.0 * e, "flops": e}
    if kind == "level":
        e = _entries(case)
        return {"bytes": 16.0 * n + 16.0 * e, "flops": e}
    if kind == "degree":
        e = 1.98 * n * case["deg"]
        return {"bytes": 16.0 * n + 8.0 * e, "flops": e}
    if kind == "color":
        e = _entries(case)
        return {"bytes": 16.0 * n + 4.0 * e, "flops": e}
    return {"bytes": 16.0 * n, "flops": float(n)}


# ------------------------------------------------------------------------------------
# the floating-point outputs in plain numpy

def _plain_phase(rowptr, tail, weight, lower: float):
    """One phase of Vite's Louvain method: all vertices move at once, each to the neighbouring
    community of largest gain (ties to the smaller id), until the modularity rises by less than
    THRESHOLD. Returns (communities, modularity, iterations)."""
    n = len(rowptr) - 1
    src = np.repeat(np.arange(n), np.diff(rowptr))
    has = np.diff(rowptr) > 0
    vdeg = np.bincount(src, weights=weight, minlength=n)
    const = 1.0 / vdeg.sum()
    loops = np.bincount(src[src == tail], weights=weight[src == tail], minlength=n)
    past, curr = np.arange(n), np.arange(n)
    cdeg, csize = vdeg.copy(), np.ones(n, np.int64)
    prev, iters = lower, 0
    while True:
        iters += 1
        keys, inv = np.unique(src * n + curr[tail], return_inverse=True)
        count = np.bincount(inv, weights=weight, minlength=len(keys))
        v, c = keys // n, keys % n
        own = c == curr[v]
        inside = np.zeros(n)
        inside[v[own]] = count[own]
        v, c, count = v[~own], c[~own], count[~own]
        eix, ax = inside - loops, cdeg[curr] - vdeg
        gain = 2.0 * (count - eix[v]) - 2.0 * vdeg[v] * (cdeg[c] - ax[v]) * const
        v, c, gain = v[gain > 0.0], c[gain > 0.0], gain[gain > 0.0]
        order = np.lexsort((c, -gain, v))
        v, c = v[order], c[order]
        first = np.ones(len(v), bool)
        first[1:] = v[1:] != v[:-1]
        target = curr.copy()
        target[v[first]] = c[first]
        stay = (csize[target] == 1) & (csize[curr] == 1) & (target > curr)
        target[stay] = curr[stay]
        moved = np.flatnonzero((target != curr) & has)
        np.add.at(cdeg, target[moved], vdeg[moved])
        np.add.at(cdeg, curr[moved], -vdeg[moved])
        np.add.at(csize, target[moved], 1)
        np.add.at(csize, curr[moved], -1)
        mod = abs(inside.sum() * const - (cdeg * cdeg).sum() * const * const)
        if math.isnan(mod) or mod - prev < THRESHOLD:
            return past, prev, iters
        prev = max(mod, lower)
        past, curr = curr, target


def _plain_coarse(rowptr, tail, weight, comm):
    """The next level's graph: communities numbered by first appearance, weights summed."""
    _, at, inv = np.unique(comm, return_index=True, return_inverse=True)
    rank = np.empty(len(at), np.int64)
    rank[np.argsort(at)] = np.arange(len(at))
    new = rank[inv]
    n = len(at)
    src = np.repeat(np.arange(len(rowptr) - 1), np.diff(rowptr))
    keys, inv = np.unique(new[src] * n + new[tail], return_inverse=True)
    out = np.zeros(n + 1, np.int64)
    out[1:] = np.cumsum(np.bincount(keys // n, minlength=n))
    return out, keys % n, np.bincount(inv, weights=weight, minlength=len(keys))


def _plain_run(graph) -> list:
    mods, last = [], -1.0
    while True:
        comm, mod, _ = _plain_phase(*graph, -1.0)
        mods.append(mod)
        if not mod - last > THRESHOLD:
            return mods
        graph, last = _plain_coarse(*graph, comm), mod


def _gini(labels) -> float:
    size = np.sort(np.bincount(labels))
    k = len(size)
    weighted = float((np.arange(1, k + 1) * size).sum())
    return 2.0 * weighted / (k * float(size.sum())) - (k + 1) / k


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "degree":
        rowptr, weight = _degree_input(case, seed)
        vdeg = torch.segment_reduce(torch.from_numpy(weight), "sum", offsets=torch.from_numpy(rowptr),
                                    initial=0.0).numpy()
        return {"vdeg": vdeg, "constant": 1.0 / math.fsum(vdeg)}
    if kind == "compare":
        truth, found = _compare_input(case, seed)

        def pairs(x):
            return int((x * (x - 1) // 2).sum())

        _, joint = np.unique(truth * (found.max() + 1) + found, return_counts=True)
        both, in1, in2 = pairs(joint), pairs(np.bincount(truth)), pairs(np.bincount(found))
        p, r = both / in2, both / in1
        return {"n": None, "nc1": None, "nc2": None, "same_same": None, "same_diff": None,
                "diff_same": None, "precision": p, "recall": r, "fscore": 2.0 * p * r / (p + r),
                "gini1": _gini(truth), "gini2": _gini(found)}
    if kind not in ("run", "level") or case["n"] >= HOST_VERTICES or _entries(case) > EXACT_ENTRIES:
        return None
    if any(case.get(k) for k in ("coloring", "vertex_order", "et_type", "threshold_scaling")):
        return None
    graph = _host_graph(case, seed)
    if kind == "run":
        return {"nv": None, "ne": None, "iters": None, "num_colors": None, "comm": None,
                "modularity": _padded(_plain_run(graph), LEVELS, np.float64)}
    comm, modularity, _ = _plain_phase(*graph, -1.0)
    coarse = _plain_coarse(*graph, comm)
    _, modularity2, _ = _plain_phase(*coarse, -1.0)
    rowptr, _, weight = coarse
    vdeg = np.bincount(np.repeat(np.arange(len(rowptr) - 1), np.diff(rowptr)), weights=weight,
                       minlength=len(rowptr) - 1)
    return {"comm": None, "modularity": modularity, "iters": None, "constant": 1.0 / vdeg.sum(),
            "vdeg": _padded(vdeg, case["n"], np.float64), "comm2": None,
            "modularity2": modularity2, "iters2": None}
