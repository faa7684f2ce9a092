"""Measured cases: the calls that programs built on this framework make, over the range of sizes they make them at.

Four kinds of work, one per public entry point:

  forward   a batch that is already on the GPU through S2VInference.forward (a serving or scoring loop that keeps its
            batches resident); `loss` adds the loss / accuracy tail of an evaluation loop on the same stream
  csr       a batch whose CSR arrays lie in pinned host memory through S2VInference.infer_host: upload, forward, download
  edges     a batch as a raw edge list in pinned host memory through Context.infer_edges_host: upload, CSR built on the
            device, forward, download; `lanes` = 2 keeps two batches in flight (submit / submit / wait / wait)
  level     one message-passing level on a single large graph through Context.level

and four families of graphs:

  molecule  random spanning tree plus 10 % extra edges (about 2.2 neighbours per node), one graph after another
  protein   random geometric graphs with about 7.4 neighbours per node, 100 to 620 nodes
  er        directed Erdos-Renyi: uniform sources and destinations
  rmat      symmetrised, deduplicated R-MAT (0.57, 0.19, 0.19, 0.05): a power law with hub rows

Everything is computed in fp32, the only data type of the path.  Inputs are made on the GPU from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from graphnn_b200 import capi, engine, giant

_STREAM = None


def listed():
    return [
        # the smallest configuration as a scoring loop meets it: 64 graphs, launches and host work are everything
        _batch("forward_mutag_64", "forward", "molecule", 64, 10, 28, tags=7, d=64, levels=3, hidden=128),
        # the same batch from host buffers, as one blocking call of a service answers a request
        _batch("csr_host_mutag_64", "csr", "molecule", 64, 10, 28, tags=7, d=64, levels=3, hidden=128),
        # an ordinary mini-batch of molecules
        _batch("forward_molecules_700", "forward", "molecule", 700, 20, 40, tags=82, d=128, levels=4, hidden=256),
        # one GPU's share of a batch that is sharded over four, not a round number
        _batch("forward_molecules_4093", "forward", "molecule", 4093, 20, 40, tags=82, d=128, levels=4, hidden=256),
        # the headline batch
        _batch("forward_molecules_16k", "forward", "molecule", 16384, 20, 40, tags=82, d=128, levels=4, hidden=256),
        # continuous node attributes instead of tags: the input projection is a real product; narrow embeddings
        _batch("forward_dense_attr_601", "forward", "molecule", 601, 18, 60, tags=21, d=32, levels=3, hidden=64, classes=6, dense=True),
        # the large batch of the protein configuration
        _batch("forward_proteins_4k", "forward", "protein", 4096, 100, 620, tags=3, d=64, levels=5, hidden=128),
        # an evaluation loop: averaged messages and mean pooling, node embeddings kept, loss and accuracy on top
        _batch("eval_proteins_301", "forward", "protein", 301, 100, 620, tags=3, d=64, levels=5, hidden=128, average=True,
               embed=True, loss=True),
        # the headline batch end to end: raw edge list on the host in, logits on the host out
        _batch("edges_host_molecules_16k", "edges", "molecule", 16384, 20, 40, tags=82, d=128, levels=4, hidden=256),
        # a serving loop with two batches in flight (one pass = two batches)
        _batch("edges_two_lanes_molecules_2048", "edges", "molecule", 2048, 20, 40, tags=82, d=128, levels=4, hidden=256, lanes=2),
        # a single large graph, uniform degrees
        _level("level_er_1m", "er", nodes=1 << 20, edges=1 << 23, d=64, x=True),
        # a single large graph with hubs
        _level("level_rmat_20", "rmat", nodes=1 << 20, edges=1 << 24, d=128, x=False),
    ]


def draw(rng):
    """One more case; sizes log-uniform, odd ones among them, none beyond the listed sizes of its family."""
    kind = rng.choice(["forward", "forward", "forward", "forward", "csr", "edges", "edges", "level", "level"])
    if kind == "level":
        d = rng.choice([32, 64, 64, 128, 128])
        if rng.random() < 0.5:
            n = _log_int(rng, 3000, (1 << 20) * 64 // max(d, 64))
            return _level(None, "er", nodes=n, edges=int(n * rng.uniform(2.0, 8.0)), d=d, x=rng.random() < 0.7, val=rng.random() < 0.3)
        scale = rng.randint(13, 20)
        return _level(None, "rmat", nodes=1 << scale, edges=int((1 << scale) * rng.uniform(4.0, 16.0)), d=d, x=scale < 20 and rng.random() < 0.3)
    classes = rng.choice([2, 2, 2, 3, 6])
    flags = {"average": rng.random() < 0.2, "embed": False, "loss": False, "dense": False, "lanes": 1}
    if kind == "forward":
        flags["embed"] = rng.random() < 0.25
        flags["loss"] = rng.random() < 0.25
        flags["dense"] = rng.random() < 0.15
    elif kind == "edges":
        flags["average"] = False   # the edge-list entry builds unit weights; its pooling follows the model
        flags["lanes"] = rng.choice([1, 2])
    if rng.random() < 0.3:
        graphs = _log_int(rng, 8, 2048 if flags["lanes"] == 2 else 4096)
        return _batch(None, kind, "protein", graphs, 100, 620, tags=3, d=rng.choice([64, 64, 64, 32, 128]) if graphs < 1000 else 64,
                      levels=rng.randint(2, 5), hidden=rng.choice([64, 128]), classes=classes, **flags)
    lo, hi = rng.choice([(10, 28), (20, 40), (20, 40), (18, 60), (2, 100)])
    most = 16384 * 40 // hi // flags["lanes"]
    return _batch(None, kind, "molecule", _log_int(rng, 8, most), lo, hi, tags=rng.choice([7, 37, 82]) if not flags["dense"] else rng.choice([3, 18, 21, 37]),
                  d=rng.choice([32, 64, 64, 128, 128]), levels=rng.randint(2, 4), hidden=rng.choice([64, 128, 256]), classes=classes, **flags)


def prepare(case, seed):
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    torch.cuda.set_stream(_STREAM)   # one stream for the library's work and torch's allocations, as in a user's loop
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 11)
    if case["kind"] == "level":
        return _prepare_level(case, seed, gen)
    d, hidden, classes = case["d"], case["hidden"], case["classes"]
    std = 0.1 if d <= 64 and case["family"] == "molecule" else 0.05
    w = {"w_n2l": (case["tags"], d), "p_node_conv": (d, d), "h1_weight": (d, hidden), "h2_weight": (hidden, classes)}
    weights = {k: (torch.randn(s, generator=gen, device="cuda") * std).cpu().numpy() for k, s in w.items()}
    state = {"case": case, "stream": _STREAM.cuda_stream,
             "eng": engine.S2VInference(weights, case["levels"], device=0, pool_average=case["average"])}
    if case["kind"] == "forward":
        b = _graphs(case, gen)
        val = None
        if case["average"]:
            deg = (b["row_ptr"][1:] - b["row_ptr"][:-1]).float()
            val = torch.repeat_interleave(1.0 / deg.clamp(min=1), deg.long())
        state["batch"] = engine.DeviceBatch(b["graphs"], b["nodes"], b["row_ptr"], b["col_idx"], b["graph_ptr"], b["tags"], b["x"], val, b["largest"])
        if case["loss"]:
            g = b["graphs"]
            state["label_ptr"] = torch.arange(g + 1, dtype=torch.int32, device="cuda")
            state["label"] = torch.randint(0, classes, (g,), generator=gen, device="cuda").to(torch.int32)
            state["one"] = torch.ones(g, device="cuda")
        return state
    hosts = []
    for _ in range(case["lanes"]):
        b = _graphs(case, gen)
        logits, pred = np.zeros((b["graphs"], classes), np.float32), np.zeros(b["graphs"], np.int32)
        pin = {k: _pinned(b[k]) for k in ("row_ptr", "col_idx", "edge_src", "edge_dst", "graph_ptr", "tags")}
        if case["kind"] == "csr":
            hb = engine.HostBatch(b["graphs"], b["nodes"], pin["row_ptr"], pin["col_idx"], pin["graph_ptr"], pin["tags"], b["largest"])
            hosts.append((hb, logits, pred))
        else:
            hosts.append((b["graphs"], b["nodes"], pin["edge_src"], pin["edge_dst"], pin["graph_ptr"], pin["tags"], logits, pred))
    state["hosts"] = hosts
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "level":
        return state["ctx"].level(*state["args"], stream=state["stream"])
    eng = state["eng"]
    if case["kind"] == "forward":
        logits, probs, pred, embed = eng.forward(state["batch"], want_embed=case["embed"], stream=state["stream"])
        if not case["loss"]:
            return logits, probs, pred, embed
        tail = torch.empty(2, device="cuda")
        each = torch.empty(logits.shape[0], device="cuda")
        eng.ctx.loss_acc(logits, state["label_ptr"], state["label"], state["one"], tail[:1], tail[1:], each, stream=state["stream"])
        return logits, probs, pred, embed, tail, each
    if case["kind"] == "csr":
        return [eng.infer_host(*h) for h in state["hosts"]]
    if len(state["hosts"]) == 1:
        eng.ctx.infer_edges_host(eng.model, *state["hosts"][0])
    else:
        for lane, h in enumerate(state["hosts"]):
            eng.ctx.infer_edges_host_submit(lane, eng.model, *h)
        for lane in range(len(state["hosts"])):
            eng.ctx.infer_host_wait(lane)
    return [h[-2:] for h in state["hosts"]]


def work(case):
    d = case["d"]
    if case["kind"] == "level":
        n = case["nodes"]
        nnz = case["edges"] if case["family"] == "er" else 2 * 0.9 * case["edges"]   # R-MAT loses about a tenth as duplicates
        dense = n * d * 4
        return {"bytes": 4 * n + nnz * (8 if case["val"] else 4) + dense * (3 if case["x"] else 2) + 4 * d * d, "flops": 2.0 * n * d * d + nnz * d}
    g, mean = case["graphs"], (case["lo"] + case["hi"]) / 2
    n = g * mean
    e = n * 7.0 if case["family"] == "protein" else 2.2 * g * (mean - 1)
    levels, hidden, classes = case["levels"], case["hidden"], case["classes"]
    in_edges = 8 * e if case["kind"] == "edges" else 4 * n + 4 * e * (2 if case["average"] and case["kind"] == "forward" else 1)
    in_nodes = 4 * n * (case["tags"] if case["dense"] else 1)
    weights = 4 * (case["tags"] * d + d * d + d * hidden + hidden * classes)
    out = g * (4 * classes + 4) + (4 * g * classes if case["kind"] == "forward" else 0) + (4 * n * d if case["embed"] else 0)
    # one-hot inputs: the first level's product has only as many distinct rows as there are tags
    products = levels * n + n * case["tags"] / d if case["dense"] else (levels - 1) * n + case["tags"]
    flops = 2.0 * d * d * products + levels * e * d + n * d + 2.0 * g * hidden * (d + classes)
    return {"bytes": case["lanes"] * (in_edges + in_nodes + 4 * g + weights + out), "flops": case["lanes"] * flops}


def tolerance(case):
    # fp32 sums in another order, 3xTF32-grade products; a prediction can only differ where two logits tie
    return {"rel": 1e-5, "max": 1e-4, "differ": 1e-3}


def _batch(name, kind, family, graphs, lo, hi, tags, d, levels, hidden, classes=2, dense=False, average=False, embed=False, loss=False, lanes=1):
    case = {"kind": kind, "family": family, "graphs": graphs, "lo": lo, "hi": hi, "tags": tags, "d": d, "levels": levels, "hidden": hidden,
            "classes": classes, "dense": dense, "average": average, "embed": embed, "loss": loss, "lanes": lanes}
    return dict(case, name=name) if name else case


def _level(name, family, nodes, edges, d, x, val=False):
    case = {"kind": "level", "family": family, "nodes": nodes, "edges": edges, "d": d, "x": x, "val": val}
    return dict(case, name=name) if name else case


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _prepare_level(case, seed, gen):
    n, d = case["nodes"], case["d"]
    val = None
    if case["family"] == "er":
        src = torch.randint(0, n, (case["edges"],), generator=gen, device="cuda")
        dst = torch.randint(0, n, (case["edges"],), generator=gen, device="cuda")
        row_ptr, col = _csr(dst.sort(stable=True).values, src, n)   # sources are independent of the destinations
        if case["val"]:
            val = torch.rand(case["edges"], generator=gen, device="cuda") + 0.5
    else:
        shard = giant.rmat_shard_on_device(n.bit_length() - 1, case["edges"], 0, 1, torch.device("cuda", 0), seed=int(seed))
        row_ptr, col = shard.row_ptr, shard.col_idx
    H = torch.randn((n, d), generator=gen, device="cuda")
    W = torch.randn((d, d), generator=gen, device="cuda") * (0.1 if d <= 64 else 0.05)
    X = torch.randn((n, d), generator=gen, device="cuda") if case["x"] else None
    ctx = capi.Context(0)
    return {"case": case, "stream": _STREAM.cuda_stream, "ctx": ctx, "args": (row_ptr, col, val, H, W, X, torch.empty((n, d), device="cuda"))}


def _csr(rows_sorted, cols, n):
    row_ptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    row_ptr[1:] = torch.cumsum(torch.bincount(rows_sorted, minlength=n), 0)
    return row_ptr, cols.to(torch.int32)


def _graphs(case, gen):
    """A block-diagonal batch on the GPU: CSR, edge list in AddEdge order, graph ranges, tags or attributes."""
    g, lo, hi = case["graphs"], case["lo"], case["hi"]
    # node counts uniform over [lo, hi] in a random order; their total does not depend on the seed
    sizes = (lo + torch.arange(g, device="cuda") % (hi - lo + 1))[torch.randperm(g, generator=gen, device="cuda")]
    off = torch.zeros(g + 1, dtype=torch.int64, device="cuda")
    off[1:] = torch.cumsum(sizes, 0)
    n = int(off[-1])
    if case["family"] == "molecule":
        graph = torch.repeat_interleave(torch.arange(g, device="cuda"), sizes)
        local = torch.arange(n, device="cuda") - off[graph]
        child = torch.nonzero(local > 0).flatten()
        first = off[graph[child]]
        parent = first + torch.minimum((torch.rand(child.shape[0], generator=gen, device="cuda") * local[child]).long(), local[child] - 1)
        extra = torch.where(sizes > 2, (sizes + 8) // 10, 0)   # a tenth of the n - 1 tree edges, rounded up
        eg = torch.repeat_interleave(torch.arange(g, device="cuda"), extra)
        m = sizes[eg]
        a = torch.minimum((torch.rand(eg.shape[0], generator=gen, device="cuda") * m).long(), m - 1)
        step = 1 + torch.minimum((torch.rand(eg.shape[0], generator=gen, device="cuda") * (m - 1)).long(), m - 2)
        u = torch.cat([parent, off[eg] + a])
        v = torch.cat([child, off[eg] + (a + step) % m])
        key = torch.unique(torch.cat([u * n + v, v * n + u]))   # both directions, sorted by (source, neighbour)
        src, dst = key // n, key % n
    else:
        points = torch.rand((g, hi, 3), generator=gen, device="cuda")
        r2 = (7.4 * 3.0 / (4.0 * math.pi * sizes.float())) ** (2.0 / 3.0)
        at = torch.arange(hi, device="cuda")
        parts = []
        for c in range(0, g, 128):
            p, s = points[c:c + 128], sizes[c:c + 128]
            d2 = sum((p[:, :, None, k] - p[:, None, :, k]) ** 2 for k in range(3))
            valid = at[None, :] < s[:, None]
            close = (d2 < r2[c:c + 128, None, None]) & valid[:, :, None] & valid[:, None, :] & (at[:, None] != at[None, :])
            gi, i, j = torch.nonzero(close, as_tuple=True)
            parts.append(torch.stack([off[c + gi] + i, off[c + gi] + j]))
        src, dst = torch.cat(parts, 1)
    row_ptr, col_idx = _csr(src, dst, n)   # the matrix is symmetric: row y lists its neighbours ascending either way
    rank_weight = 1.0 / torch.arange(1, case["tags"] + 1, device="cuda").double() ** 1.2   # Zipf tags, as atom types are
    if case["family"] == "protein" or case["tags"] < 10:
        rank_weight = torch.ones_like(rank_weight)
    tags = x = None
    if case["dense"]:
        x = torch.randn((n, case["tags"]), generator=gen, device="cuda")
    else:
        cum = torch.cumsum(rank_weight / rank_weight.sum(), 0)
        tags = torch.searchsorted(cum, torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)).clamp(max=case["tags"] - 1).to(torch.int32)
    return {"graphs": g, "nodes": n, "row_ptr": row_ptr, "col_idx": col_idx, "edge_src": src.to(torch.int32), "edge_dst": dst.to(torch.int32),
            "graph_ptr": off.to(torch.int32), "tags": tags, "x": x, "largest": int(sizes.max())}
