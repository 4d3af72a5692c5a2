"""The work that users of graphbrew_gb300 have it do, as cases that can be timed.

The package orders the vertices of a graph so that later kernels run faster on
it (the algorithm-12 mapping), rebuilds the graph in that order, runs the
kernels that such a mapping is made for, and trains the selector that decides
whether a mapping pays.  The listed cases cover these in the proportions in
which they are used: six whole mappings from the smallest graph of the tests to
the largest of the benchmark configurations, one more through host buffers as
the GAPBS builder calls the library, one order over communities that are
already known, the selector's cheap arm (DBG and a relabel), the three kernels
after a mapping, a batch of small graphs, and the selector's training.

Graphs are the seeded families of graphbrew_gb300.graphgen; every seed is
another graph.  The rebuilt graph is written to buffers that the program holds,
through the C entry points (include/gbgpu.h), as the GAPBS builder does it; their
size is that of the drawn edge list, of which duplicate edges are left out.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import graphbrew_gb300 as gb
from graphbrew_gb300 import graphgen as gg
from graphbrew_gb300 import selector

RECIPE = gb.DEFAULT_RECIPE
PARTS = RECIPE.split(":")


def _recipe(intra: str) -> str:
    return ":".join(intra if p.startswith("intra_") else p for p in PARTS)


def listed():
    return [
        # The smallest graph of the tests: a call's launches and latency.
        {"name": "map_rmat12", "do": "map", "family": "rmat", "scale": 12, "degree": 16, "host": False},
        # The first benchmark configuration (65,536 vertices, edge factor 16), through
        # host arrays as the GAPBS builder holds them: copies both ways are in the call.
        {"name": "map_rmat16_host", "do": "map", "family": "rmat", "scale": 16, "degree": 16, "host": True},
        # A graph with communities, of the sizes that the batched configuration has; an
        # odd vertex count.
        {"name": "map_planted_300k", "do": "map", "family": "planted", "n": 300007, "communities": 37, "degree": 17,
         "mixing": 0.15, "host": False},
        # A road-like graph: high diameter, neighbours at nearby ids.
        {"name": "map_grid_300k", "do": "map", "family": "grid", "rows": 511, "cols": 601, "deleted": 0.05,
         "host": False},
        # The headline configuration: scale 22, edge factor 16.
        {"name": "map_rmat22", "do": "map", "family": "rmat", "scale": 22, "degree": 16, "host": False},
        # The largest configuration: uniform random, 8M vertices, weak communities.
        {"name": "map_uniform23", "do": "map", "family": "uniform", "scale": 23, "degree": 16, "host": False},
        # Another order within communities that are already known: what a program does
        # that tries several orders on one community detection.
        {"name": "compose_rcm_rmat19", "do": "compose", "family": "rmat", "scale": 19, "degree": 13,
         "intra": "intra_rcm"},
        # The selector's cheap arm: DBG and a relabel.
        {"name": "dbg_rmat21", "do": "dbg", "family": "rmat", "scale": 21, "degree": 15},
        # The kernels after a mapping (PageRank, BFS, connected components), on a skewed
        # graph of low diameter and on a road-like one.
        {"name": "kernels_rmat20", "do": "kernels", "family": "rmat", "scale": 20, "degree": 16},
        {"name": "kernels_grid_500k", "do": "kernels", "family": "grid", "rows": 517, "cols": 1023, "deleted": 0.1},
        # Many small graphs in one call, with the library's default schedule.
        {"name": "batch_16", "do": "batch", "count": 16, "n_min": 10000, "n_max": 300000},
        # The selector's training: the whole set's 12,000 rows, a few of its epochs.
        {"name": "train_12000", "do": "train", "rows": 12000, "epochs": 4, "batch": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, n_min, n_max, families):
    """A family and its sizes: n_min..n_max vertices, spread over the logarithm."""
    family = rng.choice(families)
    n = _log(rng, n_min, n_max)
    scale = max(10, min(int(math.log2(n_max)), int(round(math.log2(n)))))
    if family == "rmat":
        return {"family": family, "scale": scale, "degree": rng.randint(4, 16)}
    if family == "uniform":
        return {"family": family, "scale": scale, "degree": rng.randint(2, 16)}
    if family == "grid":
        n = min(n, 400000)
        rows = max(16, int(math.sqrt(n) * rng.uniform(0.5, 1.5)))
        return {"family": family, "rows": rows, "cols": max(16, n // rows), "deleted": round(rng.uniform(0.0, 0.2), 3)}
    return {"family": family, "n": n, "communities": rng.randint(4, 64), "degree": rng.randint(4, 24),
            "mixing": round(rng.uniform(0.02, 0.3), 3)}


def draw(rng):
    kind = rng.choice(["map"] * 6 + ["compose", "dbg", "kernels", "kernels", "batch", "train"])
    if kind == "map":
        families = ["rmat", "rmat", "uniform", "grid", "planted"]
        return {"do": kind, **_draw_graph(rng, 1 << 12, 1 << 22, families), "host": rng.random() < 0.2}
    if kind == "compose":
        # Grids, with their thousands of levels, stay with the mapping and kernel cases.
        intra = rng.choice(["intra_rcm", "intra_gorder", "intra_bfs", "intra_hubsort"])
        return {"do": kind, **_draw_graph(rng, 1 << 14, 1 << 20, ["rmat", "planted", "uniform"]), "intra": intra}
    if kind == "dbg":
        return {"do": kind, **_draw_graph(rng, 1 << 14, 1 << 22, ["rmat", "uniform", "grid", "planted"])}
    if kind == "kernels":
        return {"do": kind, **_draw_graph(rng, 1 << 14, 1 << 21, ["rmat", "uniform", "grid", "planted"])}
    if kind == "batch":
        return {"do": kind, "count": rng.randint(4, 24), "n_min": 10000, "n_max": _log(rng, 30000, 300000)}
    return {"do": "train", "rows": rng.randint(600, 12000), "epochs": rng.randint(1, 4),
            "batch": rng.choice([32, 64, 100, 128, 256])}


def _graph(case, seed, device="cuda"):
    family = case["family"]
    if family == "rmat":
        return gg.rmat(case["scale"], case["degree"], seed=seed, device=device)
    if family == "uniform":
        return gg.uniform(case["scale"], case["degree"], seed=seed, device=device)
    if family == "grid":
        return gg.grid(case["rows"], case["cols"], case["deleted"], seed=seed, device=device)
    rp, col, _ = gg.planted_partition(case["n"], case["communities"], case["degree"], case["mixing"], seed=seed,
                                      device=device)
    return rp, col


def _batch_specs(case):
    """The sizes of a batch: log-uniform, RMAT and planted graphs in turn."""
    rng = np.random.default_rng(case["count"] * 1000003 + case["n_max"])
    specs = []
    for i in range(case["count"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        if i % 2 == 0:
            specs.append({"family": "rmat", "scale": int(math.log2(n)), "degree": int(rng.integers(8, 17))})
        else:
            specs.append({"family": "planted", "n": n, "communities": int(rng.integers(4, 65)),
                          "degree": int(rng.integers(8, 25)), "mixing": float(rng.uniform(0.05, 0.3))})
    return specs


def _rows(case, seed):
    """Rows of the selector's training set: standardised features of 12 columns (the
    kernel's three flags and the reuse count among them) and the log10 times of three arms."""
    rng = np.random.default_rng(seed)
    rows = case["rows"]
    size = rng.uniform(4.2, 6.0, rows)
    kernel = rng.integers(0, 3, rows)
    x = np.zeros((rows, 12))
    x[:, 0] = size
    x[:, 1] = size + rng.uniform(0.6, 1.8, rows)
    x[:, 2] = 10.0 ** (x[:, 1] - x[:, 0])
    x[:, 3] = rng.lognormal(0.0, 1.0, rows)
    x[:, 4:7] = rng.random((rows, 3))
    x[:, 7] = 10.0 ** size / 1.6e7
    x[np.arange(rows), 8 + kernel] = 1.0
    x[:, 11] = rng.integers(1, 3, rows)
    work = x[:, 1] - 5.0 + 0.3 * kernel
    t = np.stack([0.6 + 0.8 * work, 0.9 * work + 0.1 * np.log10(1.0 + x[:, 3]), work + 0.2 * x[:, 5]], axis=1)
    t += rng.normal(0.0, 0.05, t.shape)
    x = (x - x.mean(0)) / (x.std(0) + 1e-9)
    return x.astype(np.float32), t.astype(np.float32)


def prepare(case, seed):
    do = case["do"]
    ctx = gb.default_context()
    state = {"do": do, "ctx": ctx}
    if do == "batch":
        state["graphs"] = [_graph(s, seed * 1009 + i) for i, s in enumerate(_batch_specs(case))]
        return state
    if do == "train":
        state["x"], state["t"] = _rows(case, seed)
        state["params"] = selector.init_params(ctx, 12, seed)
        state["epochs"], state["batch"], state["seed"] = case["epochs"], case["batch"], seed
        return state
    rp, col = _graph(case, seed)
    n, device = rp.numel() - 1, "cuda"
    if case.get("host"):
        rp, col, device = rp.cpu(), col.cpu(), "cpu"
    state["rp"], state["col"] = rp, col
    if do in ("map", "dbg"):
        state["flags"] = 0 if case.get("host") else gb.DEVICE_POINTERS
        state["out"] = {"ids": torch.zeros(n, dtype=torch.int32, device=device),
                        "row_ptr": torch.zeros(n + 1, dtype=torch.int64, device=device),
                        "col": torch.zeros(max(_sizes(case)[1], col.numel()), dtype=torch.int32, device=device)}
        if do == "dbg":
            state["out"]["old"] = torch.zeros(n, dtype=torch.int32, device=device)
    if do == "compose":
        state["recipe"] = _recipe(case["intra"])
        state["members"], _ = ctx.run_graphbrew(rp, col, RECIPE)
    if do == "kernels":
        state["source"] = int(torch.argmax(rp[1:] - rp[:-1]).item())
    torch.cuda.synchronize()
    return state


def _check(ctx, status):
    if status != gb.OK:
        raise RuntimeError(gb.library().gbgpu_last_error(ctx.handle).decode())


def run(state):
    do, ctx = state["do"], state["ctx"]
    if do == "train":
        params, loss = ctx.mlp_train(state["params"], state["x"], state["t"], epochs=state["epochs"],
                                     batch=state["batch"], lr=2e-3, seed=state["seed"])
        return {"params": params, "loss": np.float32(loss)}
    if do == "batch":
        return ctx.generate_mappings_batched(state["graphs"], RECIPE)[0]
    rp, col = state["rp"], state["col"]
    if do == "map":
        out, stats = state["out"], gb.GbgpuStats()
        _check(ctx, gb.library().gbgpu_map_and_relabel(
            ctx.handle, rp.data_ptr(), col.data_ptr(), rp.numel() - 1, col.numel(), RECIPE.encode(), -1.0,
            out["ids"].data_ptr(), out["row_ptr"].data_ptr(), out["col"].data_ptr(), ctypes.byref(stats),
            state["flags"]))
        return out
    if do == "compose":
        return ctx.order_compose(rp, col, state["members"], state["recipe"])[0]
    if do == "dbg":
        out, lib = state["out"], gb.library()
        graph = (ctx.handle, rp.data_ptr(), col.data_ptr(), rp.numel() - 1, col.numel())
        _check(ctx, lib.gbgpu_dbg_mapping(*graph, out["ids"].data_ptr(), None, state["flags"]))
        _check(ctx, lib.gbgpu_relabel_csr(*graph, out["ids"].data_ptr(), out["row_ptr"].data_ptr(),
                                          out["col"].data_ptr(), out["old"].data_ptr(), state["flags"]))
        return out
    scores, sweeps, _ = ctx.pagerank(rp, col)
    depth, _ = ctx.bfs(rp, col, state["source"])
    comp, _ = ctx.connected_components(rp, col)
    return {"scores": scores, "sweeps": sweeps, "depth": depth, "comp": comp}


def _sizes(case):
    """Vertices and directed entries, as the family draws them (duplicates not taken out)."""
    if case["family"] == "grid":
        n = case["rows"] * case["cols"]
        return n, 4 * n
    if case["family"] == "planted":
        return case["n"], case["n"] * case["degree"]
    n = 1 << case["scale"]
    return n, 2 * n * case["degree"]


def work(case):
    do = case["do"]
    if do == "train":
        layers = 12 * 64 + 64 * 64 + 64 * 3
        return {"bytes": case["rows"] * 15 * 4 + 2 * 4 * (layers + 131),
                "flops": case["epochs"] * case["rows"] * 6 * layers}
    if do == "batch":
        n = math.sqrt(case["n_min"] * case["n_max"])
        return {"bytes": case["count"] * (8 * n + 4 * 20 * n + 4 * n), "flops": 0}
    n, entries = _sizes(case)
    entries = int(entries * (1.0 - case.get("deleted", 0.0)))
    graph = 8 * (n + 1) + 4 * entries
    if do == "map":  # the graph in; the map and the graph in its order out
        return {"bytes": 2 * graph + 4 * n, "flops": 0}
    if do == "compose":  # the graph and the communities in, the map out
        return {"bytes": graph + 8 * n, "flops": 0}
    if do == "dbg":  # the graph in; the map, its inverse and the graph in its order out
        return {"bytes": 2 * graph + 8 * n, "flops": 0}
    return {"bytes": 3 * graph + 12 * n, "flops": 0}


def _exact_pagerank(rp, col):
    """The Jacobi sweeps of PageRank (damping 0.85, at most 20, until the change is below 1e-4)."""
    n = rp.numel() - 1
    degree = rp[1:] - rp[:-1]
    row = torch.repeat_interleave(torch.arange(n, device=rp.device), degree)
    col = col.long()
    score = torch.full((n,), 1.0 / n, dtype=torch.float64, device=rp.device)
    for _ in range(20):
        share = torch.where(degree > 0, score / degree.clamp(min=1), torch.zeros_like(score))
        new = torch.zeros_like(score).index_add_(0, row, share[col]) * 0.85 + 0.15 / n
        change = (new - score).abs().sum().item()
        score = new
        if change < 1e-4:
            break
    return score


def _exact_training(case, seed, params):
    """Adam on minibatches of a seeded shuffle (SplitMix64, Fisher-Yates from the back), in 64 bits."""
    x, t = _rows(case, seed)
    x, t = x.astype(np.float64), t.astype(np.float64)
    rows, batch, mask = case["rows"], case["batch"], (1 << 64) - 1
    cuts = np.cumsum([12 * 64, 64, 64 * 64, 64, 64 * 3])
    p = params.astype(np.float64)
    m, v = np.zeros_like(p), np.zeros_like(p)
    order = list(range(rows))
    word = (seed ^ 0x9E3779B97F4A7C15) & mask
    step, loss = 0, 0.0
    for _ in range(case["epochs"]):
        for i in range(rows - 1, 0, -1):
            word = (word + 0x9E3779B97F4A7C15) & mask
            z = ((word ^ (word >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (i + 1)
            order[i], order[j] = order[j], order[i]
        losses = []
        for at in range(0, rows, batch):
            pick = order[at:at + batch]
            w1, b1, w2, b2, w3, b3 = np.split(p, cuts)
            w1, w2, w3 = w1.reshape(12, 64), w2.reshape(64, 64), w3.reshape(64, 3)
            xb, tb = x[pick], t[pick]
            h1 = np.maximum(xb @ w1 + b1, 0.0)
            h2 = np.maximum(h1 @ w2 + b2, 0.0)
            d = h2 @ w3 + b3 - tb
            losses.append(np.mean(d * d))
            dy = 2.0 * d / d.size
            d2 = (dy @ w3.T) * (h2 > 0)
            d1 = (d2 @ w2.T) * (h1 > 0)
            g = np.concatenate([(xb.T @ d1).ravel(), d1.sum(0), (h1.T @ d2).ravel(), d2.sum(0), (h2.T @ dy).ravel(),
                                dy.sum(0)])
            step += 1
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            p = p - 2e-3 * (m / (1.0 - 0.9 ** step)) / (np.sqrt(v / (1.0 - 0.999 ** step)) + 1e-8)
        loss = float(np.mean(losses))
    return {"params": p, "loss": np.float64(loss)}


def exact(case, seed):
    if case["do"] == "kernels":
        rp, col = _graph(case, seed)
        return {"scores": _exact_pagerank(rp, col), "sweeps": None, "depth": None, "comp": None}
    if case["do"] == "train":
        return _exact_training(case, seed, prepare(case, seed)["params"])
    return None
