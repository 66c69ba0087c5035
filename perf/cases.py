"""Timed cases: the work a program has this library do, through its public entry points.

A case is a dict of plain values; ``op`` names the call, the other entries its
sizes. Graphs are R-MAT (a, b, c, d = .57, .19, .19, .05) or the social shape
(Chung-Lu, exponent 2.3, largest expected degree 9,000); half of a graph's
edges are loaded, as the sliding-window demo does. Updates slide a window over
the edges: every pass inserts the next ``half_batch`` edges and deletes the
oldest as many, round a cycle, so a state can be run any number of times.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import gpma_bfs_gb300 as G

SLIDES = 100  # batches a cycle holds (fewer where the graph is too small for that many)
SOCIAL = {"graph": "social", "nodes": 1632803, "edges": 30622564}
RMAT16 = {"graph": "rmat", "scale": 16, "edge_factor": 16}


def listed():
    return [
        # the smallest served update: 1,000 keys in host arrays into a resident large graph (latency)
        dict(SOCIAL, name="update_social_1k", op="update", half_batch=500, host=True),
        # the sliding-window demo's 1 % step on its small graph: recorded update + BFS, batch in pinned memory
        dict(RMAT16, name="step_rmat16", op="step", half_batch=4850),
        # the demo's step on the social graph: 306,224 keys, half inserts, half deletes, on the device
        dict(SOCIAL, name="update_social_306k", op="update", half_batch=153112, host=False),
        # the demo's first call: a new graph, then half of all edges in one batch (bulk rebuild)
        dict(SOCIAL, name="load_social", op="load"),
        # the largest batches: 10.5M keys into an R-MAT graph, more than 5M of them insertions (bulk rebuild)
        dict(name="update_rmat21_10M", op="update", graph="rmat", scale=21, edge_factor=32, half_batch=5250000,
             host=False),
        # one search of a small graph (latency)
        dict(RMAT16, name="bfs_rmat16", op="bfs"),
        # one search of the social graph
        dict(SOCIAL, name="bfs_social", op="bfs"),
        # 16 searches of the social graph at once, with levels
        dict(SOCIAL, name="bfs_multi_social_16", op="bfs_multi", sources=16),
        # many graphs per launch: 20 graphs of 10k to 2M edges, batches of 100 to 200k keys each
        dict(name="batch_update_20", op="batch_update", graphs=20),
        # many graphs per launch: 64 searches in each of 128 graphs, reached counts
        dict(name="batch_bfs_128", op="batch_bfs", graphs=128, sources=64),
        # analytics on the resident social graph
        dict(SOCIAL, name="pagerank_social", op="pagerank", iterations=20),
        dict(SOCIAL, name="components_social", op="components"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng):
    if rng.random() < 0.5:
        return {"graph": "rmat", "scale": rng.randint(10, 21), "edge_factor": rng.randint(8, 24)}
    nodes = _log_int(rng, 2000, 1632803)
    return {"graph": "social", "nodes": nodes, "edges": int(nodes * rng.uniform(8, 18.7))}


def _most_edges(case):
    return case["edges"] if case["graph"] == "social" else case["edge_factor"] << case["scale"]


def draw(rng):
    op = rng.choice(["update", "update", "update", "step", "load", "bfs", "bfs", "bfs_multi", "batch_update",
                     "batch_bfs", "pagerank", "components"])
    if op in ("batch_update", "batch_bfs"):
        case = {"op": op, "graphs": rng.randint(2, 20) if op == "batch_update" else _log_int(rng, 2, 128)}
        if op == "batch_bfs":
            case["sources"] = rng.randint(1, 64)
        return case
    case = dict(_draw_graph(rng), op=op)
    if op in ("update", "step"):
        case["half_batch"] = _log_int(rng, 1, max(2, min(500000, _most_edges(case) // 8)))
    if op == "update":
        case["host"] = rng.random() < 0.5
    if op == "bfs_multi":
        case["sources"] = rng.randint(1, 64) if _most_edges(case) < 2000000 else rng.randint(1, 16)
    if op == "pagerank":
        case["iterations"] = rng.randint(1, 40)
    return case


# ---- inputs ---------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rmat_ids(scales, gen):
    """Source and target of one R-MAT edge per entry of `scales` (bits of its node ids)."""
    src = torch.zeros_like(scales)
    dst = torch.zeros_like(scales)
    for level in range(int(scales.max())):
        r = torch.rand(len(scales), generator=gen, device="cuda")
        go = scales > level
        src = torch.where(go, (src << 1) | (r >= 0.76), src)
        dst = torch.where(go, (dst << 1) | ((r >= 0.57) & (r < 0.76)) | (r >= 0.95), dst)
    return src, dst


def _shuffled_unique(keys, gen):
    keys = torch.unique(keys)
    return keys[torch.randperm(len(keys), generator=gen, device="cuda")]


def _edges(case, gen):
    """(node count, shuffled distinct edge keys src << 32 | dst without self-loops) on the device."""
    if case["graph"] == "rmat":
        n, m = 1 << case["scale"], case["edge_factor"] << case["scale"]
        # twice the edges drawn: at least m of them are distinct (the same count whatever the seed)
        src, dst = _rmat_ids(torch.full((2 * m,), case["scale"], dtype=torch.int64, device="cuda"), gen)
        keep = src != dst
        return n, _shuffled_unique((src[keep] << 32) | dst[keep], gen)[:m]
    n, m = case["nodes"], case["edges"]
    ids = torch.arange(n, dtype=torch.float64, device="cuda")
    alpha, target = 1.0 / 1.3, min(9000.0, n / 4) * n / m
    lo, hi = 1e-3, float(n)
    for _ in range(40):
        mid = 0.5 * (lo + hi)
        w = (ids + mid) ** -alpha
        lo, hi = (mid, hi) if float(w[0] / w.mean()) > target else (lo, mid)
    cdf = torch.cumsum((ids + 0.5 * (lo + hi)) ** -alpha, 0)
    relabel = torch.randperm(n, generator=gen, device="cuda")
    pick = lambda: torch.searchsorted(  # noqa: E731
        cdf, torch.rand(m + m // 10, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]).clamp_(max=n - 1)
    src, dst = pick(), relabel[pick()]
    keep = src != dst
    return n, _shuffled_unique((src[keep] << 32) | dst[keep], gen)[:m]


class _View:
    """Library-owned device memory for torch.as_tensor; keeps the graph alive."""

    def __init__(self, owner, ptr, n, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _arrays(state, g):
    """The graph's key, value and row-offset arrays, in place."""
    at = g.device_arrays() + (g.get_size(),)
    if state.get("at") != at:
        k, v, r, size = at
        state["arrays"] = [torch.as_tensor(_View(g, k, size, "<i8"), device="cuda"),
                           torch.as_tensor(_View(g, v, size, "|u1"), device="cuda"),
                           torch.as_tensor(_View(g, r, g.row_num + 1, "<i4"), device="cuda")]
        state["at"] = at
    return state["arrays"]


def _slides(keys, half_batch, most=SLIDES, least=4):
    """(edges to load, the cycle's batches, their values): batch t inserts part t of the
    cycle and deletes the part half a cycle away, so half of the cycle is always live."""
    m = len(keys)
    h = max(1, min(half_batch, m // least))
    parts = min(most, m // h) & ~1
    ring = keys[:parts * h].view(parts, h)
    load = keys[parts * h // 2:parts * h // 2 + m // 2]
    batches = torch.cat([ring, ring.roll(-(parts // 2), 0)], 1)
    values = torch.zeros(2 * h, dtype=torch.uint8, device="cuda")
    values[:h] = 1
    return load, batches, values


def _loaded(n, keys):
    g = G.GPMA(n)
    G.update_gpma(g, keys, torch.ones(len(keys), dtype=torch.uint8, device="cuda"))
    return g


class _Step(G.Step):
    """A recorded step, closed with its state and before its graph."""

    def __del__(self):
        self.close()


def _batch_graphs(count, gen):
    """(nodes, edge keys) of `count` R-MAT graphs of 10k to 2M edges (spread by their logarithm), about edges/16 nodes."""
    u = (torch.arange(count, device="cuda", dtype=torch.float64) + 0.5) / count
    want = torch.exp(math.log(10000) + u * math.log(200)).long()
    scale = torch.log2(want / 16).round().long()
    of = torch.repeat_interleave(torch.arange(count, device="cuda"), 2 * want)  # twice, as for one graph
    src, dst = _rmat_ids(scale[of], gen)
    keep = src != dst
    key = _shuffled_unique((of[keep] << 48) | (src[keep] << 24) | dst[keep], gen)
    key = key[torch.sort(key >> 48, stable=True).indices]
    counts = torch.bincount(key >> 48, minlength=count).tolist()
    key = (((key >> 24) & 0xFFFFFF) << 32) | (key & 0xFFFFFF)
    return [(1 << s, k[:w]) for s, w, k in zip(scale.tolist(), want.tolist(), torch.split(key, counts))]


def prepare(case, seed):
    gen = _generator(seed)
    op = case["op"]
    state = {"op": op, "t": 0}
    if op in ("batch_update", "batch_bfs"):
        specs = _batch_graphs(case["graphs"], gen)
        state["graphs"] = graphs = [G.GPMA(n) for n, _ in specs]
        state["batch"] = b = G.Batch()
        rng = np.random.default_rng(seed)
        loads, slides = [], []
        for i, (_, keys) in enumerate(specs):
            # batch sizes spread over [100, 200k] by their logarithm, out of step with the graph sizes
            h = int(100 * 2000 ** (0.618034 * (i + 1) % 1)) // 2
            load, batches, values = _slides(keys, h, most=8, least=8)
            loads.append(load)
            slides.append((batches, values))
        off = np.concatenate([[0], np.cumsum([len(x) for x in loads])]).astype(np.uint64)
        b.update_packed(graphs, torch.cat(loads), torch.ones(int(off[-1]), dtype=torch.uint8, device="cuda"), off)
        if op == "batch_bfs":
            state["sources"] = []
            for load in loads:
                src = torch.unique(load >> 32).cpu().numpy().astype(np.uint32)
                state["sources"].append(rng.choice(src, min(case["sources"], len(src)), replace=False))
            return state
        state["views"] = [{} for _ in graphs]
        state["keys"] = [torch.cat([x[t] for x, _ in slides]) for t in range(8)]
        state["values"] = torch.cat([v for _, v in slides])
        state["offsets"] = np.concatenate([[0], np.cumsum([len(v) for _, v in slides])]).astype(np.uint64)
        return state
    n, keys = _edges(case, gen)
    state.update(n=n, m=len(keys))
    if op == "load":
        state["keys"] = keys[:len(keys) // 2].clone()
        state["values"] = torch.ones(len(state["keys"]), dtype=torch.uint8, device="cuda")
        return state
    if op in ("update", "step"):
        load, batches, values = _slides(keys, case["half_batch"])
        state["g"] = g = _loaded(n, load)
        if op == "step":
            host = batches.cpu().pin_memory()
            state["keys"], state["values"] = list(host.unbind(0)), values.cpu().pin_memory()
            state["step"] = _Step(g)
            state["levels"] = torch.zeros(n, dtype=torch.int32, device="cuda")
            state["source"] = int(load[0] >> 32)
        elif case["host"]:
            state["keys"], state["values"] = list(batches.cpu().numpy().view(np.uint64)), values.cpu().numpy()
        else:
            state["keys"], state["values"] = list(batches.unbind(0)), values
        return state
    load = keys[:len(keys) // 2]
    state["g"] = _loaded(n, load)
    if op == "bfs":
        state["sources"] = (load[:8] >> 32).tolist()
        state["levels"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    elif op == "bfs_multi":
        state["sources"] = np.resize(torch.unique(load[:256] >> 32).cpu().numpy().astype(np.uint32), case["sources"])
        state["levels"] = torch.zeros((case["sources"], n), dtype=torch.int32, device="cuda")
    elif op == "pagerank":
        state["iterations"] = case["iterations"]
        state["out"] = torch.zeros(n, dtype=torch.float32, device="cuda")
    else:
        state["out"] = torch.zeros(n, dtype=torch.int32, device="cuda")
    return state


# ---- one pass ---------------------------------------------------------------------

def run(state):
    op, t = state["op"], state["t"]
    state["t"] = t + 1
    if op == "update":
        g = state["g"]
        G.update_gpma(g, state["keys"][t % len(state["keys"])], state["values"])
        return _arrays(state, g)
    if op == "step":
        g = state["g"]
        reached = state["step"].run(state["keys"][t % len(state["keys"])], state["values"], state["source"],
                                    state["levels"])
        return [state["levels"], reached] + _arrays(state, g)
    if op == "load":
        g = G.GPMA(state["n"])
        G.update_gpma(g, state["keys"], state["values"])
        return _arrays({}, g)  # the views keep the graph
    if op == "bfs":
        return list(G.gpma_bfs(state["g"], state["n"], state["m"], state["sources"][t % 8], state["levels"]))
    if op == "bfs_multi":
        return list(G.gpma_bfs_multi(state["g"], state["sources"], state["levels"]))
    if op == "batch_update":
        state["batch"].update_packed(state["graphs"], state["keys"][t % len(state["keys"])], state["values"],
                                     state["offsets"])
        return [_arrays(view, g) for view, g in zip(state["views"], state["graphs"])]
    if op == "batch_bfs":
        return np.concatenate(state["batch"].bfs_multi(state["graphs"], state["sources"])[1])
    if op == "pagerank":
        return list(G.pagerank(state["g"], iterations=state["iterations"], out=state["out"]))
    labels, count, rounds = G.components(state["g"], out=state["out"])
    return [labels, count]


# ---- what a pass cannot do without ------------------------------------------------

def work(case):
    op = case["op"]
    if op == "batch_update":
        keys = 26000 * case["graphs"]  # mean of a log-uniform batch
        return {"bytes": 9 * keys + 18 * 16 * keys // 2, "flops": 0}
    if op == "batch_bfs":
        edges = 187000 * case["graphs"]  # mean of half the edges of a graph
        return {"bytes": 9 * edges + 8 * edges // 16, "flops": 0}
    n = case["nodes"] if case["graph"] == "social" else 1 << case["scale"]
    live = _most_edges(case) // 2
    if op == "load":
        return {"bytes": 9 * live + 9 * (live + n) + 4 * n, "flops": 0}
    if op in ("update", "step"):
        # the batch, and the leaf segment of every insertion read and written (all of the array at most)
        h = min(case["half_batch"], live // 2)
        moved = 18 * h + h + min(18 * 32 * h, 18 * (live + n))
        return {"bytes": moved + (9 * live + 8 * n if op == "step" else 0), "flops": 0}
    if op == "bfs":
        return {"bytes": 9 * live + 8 * n, "flops": 0}
    if op == "bfs_multi":
        return {"bytes": 9 * live + 4 * n + 4 * n * case["sources"], "flops": 0}
    if op == "pagerank":
        return {"bytes": 9 * live + 4 * n, "flops": 2 * live * case["iterations"]}
    return {"bytes": 9 * live + 4 * n, "flops": 0}


def exact(case, seed):
    """PageRank in 64 bits; the other cases return whole numbers."""
    if case["op"] != "pagerank":
        return None
    n, keys = _edges(case, _generator(seed))
    keys = keys[:len(keys) // 2]
    src, dst = keys >> 32, keys & 0xFFFFFFFF
    deg = torch.bincount(src, minlength=n).double()
    rank = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    for _ in range(case["iterations"]):
        share = torch.where(deg > 0, rank / deg.clamp(min=1), 0.0)
        dangling = rank[deg == 0].sum()
        rank = 0.15 / n + 0.85 * (torch.zeros_like(rank).index_add_(0, dst, share[src]) + dangling / n)
    return [rank, None]
