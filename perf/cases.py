"""Performance cases: what a user of this framework has it do, through its public entry points.

Every case is a dict of plain values with an ``op``:

  spmm       ``core.spmm_tc`` and ``core.spmm_transpose`` on the arrays of one graph: one forward and
             one transposed product, what a graph convolution's forward and backward pass ask for
  build      a new CSR graph on the GPU becomes a ``BCSRGraph`` and its transposed graph
  sample     ``BCSRSampler.sample_layers``: the per-hop blocks of one mini-batch
  infer      ``GCN_BCSR.inference``: the forward pass over a whole graph
  epoch      one full-graph training step (``train_step_full``, or captured: ``graphed_full_step``)
  sampled    one sampled training step (``train_step_sampled``, or captured: ``graphed_sampled_step``)

Graphs are seeded power-law and planted-community graphs with self-loops and symmetric normalisation,
of the shapes the benchmark has.  ``edges`` counts undirected pairs: a graph has
``2 * edges + nodes`` entries.  Models run without dropout so that their results can be compared.
"""
import math

import numpy as np
import torch

from graph_rws_b200 import BCSRGraph, GCN_BCSR, core
from graph_rws_b200.data import CSRTopology
from graph_rws_b200.helper import graphed_full_step, graphed_sampled_step, train_step_full, train_step_sampled
from graph_rws_b200.sampler import BCSRSampler

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
ESIZE = {"f32": 4, "f16": 2, "bf16": 2}
COMMUNITIES = 50
INTRA = 0.8


def listed():
    return [
        # a layer of a small citation graph in the default storage type: launch latency and host path
        dict(name="spmm_small_f32", op="spmm", graph="power", nodes=2708, edges=5278, width=16, dtype="f32"),
        # class-wide product (47 classes) of a ragged graph: a width that is no multiple of 8
        dict(name="spmm_odd_f32", op="spmm", graph="power", nodes=53777, edges=400003, width=47, dtype="f32"),
        # the SpMM microbenchmark: mid-size graph, 128 features, half precision
        dict(name="spmm_mid_f16", op="spmm", graph="power", nodes=169343, edges=1166243, width=128, dtype="f16"),
        # the same in fp32, the default storage type of graphs and of the operators
        dict(name="spmm_mid_f32", op="spmm", graph="power", nodes=169343, edges=1166243, width=128, dtype="f32"),
        # hidden-width product of the dense-community graph, the largest graph trained in full
        dict(name="spmm_dense_bf16", op="spmm", graph="community", nodes=232965, edges=57183517, width=256, dtype="bf16"),
        # a graph is loaded or has changed: both directions of it are built
        dict(name="build_mid_f32", op="build", graph="power", nodes=169343, edges=1166243, dtype="f32"),
        # inference on a handful of nodes: two hops, latency
        dict(name="sample_few", op="sample", nodes=169343, edges=1166243, seeds=37, fanouts="10,5", dtype="f32", topology="bcsr"),
        # the mini-batch of sampled training: 1,024 seeds, three hops
        dict(name="sample_batch", op="sample", nodes=2449029, edges=61860000, seeds=1024, fanouts="15,10,5", dtype="f16", topology="csr"),
        # class scores of every node of the mid-size graph
        dict(name="infer_mid_f16", op="infer", graph="power", nodes=169343, edges=1166243, features=128, hidden=128, classes=40,
             dtype="f16"),
        # one epoch of the small full-batch GCN, step by step from Python
        dict(name="epoch_small", op="epoch", graph="power", nodes=2708, edges=5278, features=1440, hidden=16, classes=7, dtype="f32",
             captured=False),
        # one epoch of full-graph training on the dense-community graph, captured once and replayed
        dict(name="epoch_dense", op="epoch", graph="community", nodes=232965, edges=57183517, features=608, hidden=256, classes=41,
             dtype="bf16", captured=True),
        # one step of sampled training, sampler and training as the two branches of one captured step
        dict(name="sampled_step", op="sampled", nodes=2449029, edges=61860000, features=128, hidden=256, classes=47, seeds=1024,
             fanouts="15,10,5", dtype="f16", captured=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["spmm", "spmm", "spmm", "build", "sample", "infer", "epoch", "sampled"])
    nodes = _log(rng, 2500, 250000)
    edges = int(nodes * math.exp(rng.uniform(math.log(2.0), math.log(16.0))))
    if op in ("spmm", "build"):
        c = dict(op=op, graph="power", nodes=nodes, edges=edges, dtype=rng.choice(["f32", "f32", "f16", "bf16"]))
        if rng.random() < 0.25:                       # dense communities
            nodes = _log(rng, 10000, 120000)
            c.update(graph="community", nodes=nodes, edges=int(nodes * rng.uniform(30, 120)))
        if op == "spmm":
            c["width"] = rng.choice([8, 16, 32, 40, 41, 47, 64, 100, 128, 128, 172, 256])
        return c
    if op == "sample":
        return dict(op=op, nodes=_log(rng, 20000, 2400000), edges=0, seeds=_log(rng, 16, 2048),
                    fanouts=rng.choice(["10,5", "15,10,5", "25,10", "5,5,5", "20"]), dtype=rng.choice(["f32", "f16", "bf16"]),
                    topology="csr", degree=rng.randint(6, 25))
    if op == "infer":
        return dict(op=op, graph="power", nodes=nodes, edges=edges, features=rng.choice([64, 100, 128, 256]),
                    hidden=rng.choice([16, 64, 128, 256]), classes=rng.choice([7, 40, 41, 47]), dtype=rng.choice(["f32", "bf16", "f16"]))
    if op == "epoch":
        captured = rng.random() < 0.5
        return dict(op=op, graph="power", nodes=nodes, edges=edges, features=rng.choice([64, 100, 128, 256, 500]),
                    hidden=rng.choice([16, 64, 128, 256]), classes=rng.choice([7, 40, 41, 47]),
                    dtype=rng.choice(["f32", "bf16", "f16"]), captured=captured)
    return dict(op=op, nodes=_log(rng, 50000, 1000000), edges=0, degree=rng.randint(6, 20), features=rng.choice([64, 100, 128]),
                hidden=rng.choice([64, 128, 256]), classes=rng.choice([7, 40, 47]), seeds=rng.choice([256, 500, 1024]),
                fanouts=rng.choice(["10,5", "15,10,5", "10,10"]), dtype=rng.choice(["f32", "f16", "bf16"]), captured=rng.random() < 0.5)


def _edges(case):
    return case["edges"] or case["nodes"] * case["degree"]


def _fanouts(case):
    return [int(f) for f in case["fanouts"].split(",")]


def _rank(u, n):
    """Ranks below ``n`` drawn with weight ~ (rank + 1)^(-2/3), from uniform numbers: the power law with
    exponent 2.5.  Closed form, so that a seed gives the same graph in every process."""
    r = ((1.0 + u * ((n + 1.0) ** (1.0 / 3.0) - 1.0)) ** 3 - 1.0).floor().long()
    return torch.minimum(r, n - 1) if torch.is_tensor(n) else r.clamp_(max=n - 1)


def _csr(case, seed, device):
    """CSR (row_ptr, col_idx, values) of the case's graph: ``edges`` distinct undirected pairs, self-loops,
    weights deg^-1/2 * deg^-1/2."""
    gen = torch.Generator(device=device).manual_seed(seed)
    n, e = case["nodes"], _edges(case)

    def uniform(m):
        return torch.rand(m, generator=gen, device=device, dtype=torch.float64)

    if case.get("graph") == "community":
        bounds = torch.arange(COMMUNITIES + 1, device=device) * n // COMMUNITIES
        size = bounds[1:] - bounds[:-1]

        def pairs(m):
            cu = torch.randint(0, COMMUNITIES, (m,), generator=gen, device=device)
            cv = torch.where(uniform(m) < INTRA, cu, torch.randint(0, COMMUNITIES, (m,), generator=gen, device=device))
            return bounds[cu] + _rank(uniform(m), size[cu]), bounds[cv] + _rank(uniform(m), size[cv])
    else:
        place = torch.randperm(n, generator=gen, device=device)        # hubs anywhere among the ids

        def pairs(m):
            return place[_rank(uniform(m), n)], place[_rank(uniform(m), n)]
    got = torch.empty(0, dtype=torch.int64, device=device)
    while got.numel() < e:
        u, v = pairs(int((e - got.numel()) * 1.3) + 4096)
        keep = u != v
        key = torch.minimum(u, v) * n + torch.maximum(u, v)
        got = torch.unique(torch.cat([got, key[keep]]))
        del u, v, keep, key
    got = got[torch.randperm(got.numel(), generator=gen, device=device)[:e]]
    u, v, own = got // n, got % n, torch.arange(n, device=device)
    key = torch.cat([u * n + v, v * n + u, own * n + own]).sort().values
    del got, u, v, own
    r, c = key // n, key % n
    counts = torch.bincount(r, minlength=n)
    scale = counts.double() ** -0.5
    rp = torch.zeros(n + 1, dtype=torch.int64, device=device)
    torch.cumsum(counts, 0, out=rp[1:])
    return rp, c.int(), (scale[r] * scale[c]).float()


def _relabel(rp, ci, vv, n, gen, device):
    full = n // 16
    ids = torch.randperm(full, generator=gen, device=device).view(-1, 1) * 16 + torch.rand(
        full, 16, generator=gen, device=device).argsort(1)
    ids = torch.cat([ids.reshape(-1), torch.arange(full * 16, n, device=device)])
    rows = torch.repeat_interleave(torch.arange(n, device=device), rp[1:] - rp[:-1], output_size=ci.numel())
    key, order = torch.sort(ids[rows] * n + ids[ci.long()])
    out = torch.zeros(n + 1, dtype=torch.int64, device=device)
    torch.cumsum(torch.bincount(key // n, minlength=n), 0, out=out[1:])
    return out, (key % n).int(), vv[order].contiguous()


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    torch.manual_seed(seed)
    gen = torch.Generator(device=device).manual_seed(seed + 1)
    op, n, dtype = case["op"], case["nodes"], DTYPES[case["dtype"]]
    s = {"case": case, "n": n, "device": device, "dtype": dtype}
    if op == "build":
        # one graph, its windows and the nodes inside them relabelled at random: what is built has the same
        # sizes whatever the seed
        s["csr"] = _relabel(*_csr(case, 1002, device), n, gen, device)
        return s
    rp, ci, vv = _csr(case, seed, device)
    if op == "spmm":
        g = BCSRGraph.from_csr(n, rp, ci, vv, device=device, values_dtype=dtype)
        s["arrays"] = (g.window_offset, g.original_col_indices, g.values_condensed)
        s["H"] = torch.randn(n, case["width"], generator=gen, device=device).to(dtype)
        s["G"] = torch.randn(g.num_windows * 16, case["width"], generator=gen, device=device).to(dtype)
        return s
    if op == "sample":
        s["seeds"] = torch.randperm(n, generator=gen, device=device)[:case["seeds"]].int()
        s["sampler"] = BCSRSampler(_fanouts(case), verbose=False, seed=seed & 0xffff)
        s["graph"] = (CSRTopology(rp, ci, vv, device=device, block_dtype=dtype) if case["topology"] == "csr" else
                      BCSRGraph.from_csr(n, rp, ci, vv, device=device, values_dtype=dtype))
        return s
    captured = case.get("captured", False)
    x = torch.randn(n, case["features"], generator=gen, device=device).to(dtype)
    y = torch.randint(0, case["classes"], (n,), generator=gen, device=device)
    hops = len(_fanouts(case)) if op == "sampled" else 3 if op == "infer" else 2
    model = GCN_BCSR(case["features"], case["hidden"], case["classes"], num_layers=hops, dropout=0.0,
                     use_checkpoint=False).to(device).to(dtype)
    if op == "infer":
        s.update(graph=BCSRGraph.from_csr(n, rp, ci, vv, device=device, values_dtype=dtype), model=model.eval(), x=x)
        return s
    opt = torch.optim.Adam(model.parameters(), lr=1e-3, eps=1e-4, capturable=captured, fused=captured)
    s.update(model=model, params=list(model.parameters()))
    if op == "epoch":
        graph = BCSRGraph.from_csr(n, rp, ci, vv, device=device, values_dtype=dtype)
        idx = torch.randperm(n, generator=gen, device=device)[:n // 2].sort().values
        if captured:
            s["step"] = graphed_full_step(model, graph, x, y, idx, opt)
        else:
            s["step"] = lambda: train_step_full(model, graph, x, y, idx, opt)
        return s
    topo = CSRTopology(rp, ci, vv, device=device, block_dtype=dtype)
    sampler = BCSRSampler(_fanouts(case), verbose=False, pad_to=256, seed=seed & 0xffff)
    order = torch.randperm(n, generator=gen, device=device).int()
    k = case["seeds"]
    batches = [order[i * k:(i + 1) * k].contiguous() for i in range(8)]
    s["i"] = 0
    if captured:
        step = graphed_sampled_step(model, sampler, topo, x, y, opt, k, pipelined=True)
        step.prime(batches[7], 0)

        def one():
            s["i"] += 1
            return step(batches[s["i"] % 8], s["i"])
    else:
        def one():
            s["i"] += 1
            sampler.step = s["i"]
            return train_step_sampled(model, sampler, topo, x, y, batches[s["i"] % 8], opt)
    s["step"] = one
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "spmm":
        C, _ = core.spmm_tc(*s["arrays"], s["H"])
        D = core.spmm_transpose(*s["arrays"], s["G"], s["n"])
        return C, D
    if op == "build":
        g = BCSRGraph.from_csr(s["n"], *s["csr"], device=s["device"], values_dtype=s["dtype"])
        t = g.transposed()
        return [(h.window_offset, h.original_col_indices, h.values_condensed) for h in (g, t)]
    if op == "sample":
        blocks = s["sampler"].sample_layers(s["graph"], s["seeds"])
        return [(b.window_offset, b.original_col_indices, b.values_condensed, b.output_nodes, b.input_nodes) for b in blocks]
    if op == "infer":
        with torch.no_grad():
            return s["model"].inference(s["graph"], s["x"])
    loss = s["step"]()
    return {"loss": loss, "params": [p.detach() for p in s["params"]], "grads": [p.grad for p in s["params"]]}


def _tiles(case):
    """Expected 16x8 tiles of the graph: distinct columns of a window, each slot of a tile one of them."""
    n, e = case["nodes"], _edges(case)
    nnz, windows = 2 * e + n, (n + 15) // 16
    if case.get("graph") != "community":
        w = (np.arange(n) + 1.0) ** (-2.0 / 3.0)
        distinct = float(-np.expm1(-2.0 * e / windows * (w / w.sum())).sum()) + 16
        return windows * distinct / 8 + windows / 2
    size = max(16, n // COMMUNITIES)
    w = (np.arange(size) + 1.0) ** (-2.0 / 3.0)
    p = w / w.sum()
    total, starts = 0.0, np.linspace(0, size - 16, 32).astype(int)
    for a in starts:                                  # windows of hubs have more entries than the others
        entries = 2.0 * e / COMMUNITIES * float(p[a:a + 16].sum())
        total += float(-np.expm1(-INTRA * entries * p).sum()) + (COMMUNITIES - 1) * float(
            -np.expm1(-(1 - INTRA) * entries / (COMMUNITIES - 1) * p).sum())
    return windows * min(total / len(starts), nnz / windows) / 8 + windows / 2


def _graph_bytes(case):
    return 8 * (case["nodes"] // 16 + 2) + _tiles(case) * (32 + 128 * ESIZE[case["dtype"]])


def _hops(case):
    """(destination rows, slots of the neighbour lists) per hop."""
    d, out = case["seeds"], []
    pad = 256 if case["op"] == "sampled" else 1
    for f in reversed(_fanouts(case)):
        out.append((d, d * f))
        d = -(-d * (1 + f) // pad) * pad
    return out


def _sampling_bytes(case):
    """Row offsets of the frontier, the drawn neighbours with their weights, the source lists and the blocks.
    Frontiers reach their bound only where no node is drawn twice; half of it is what graphs like these give."""
    total, v = 0.0, ESIZE[case["dtype"]]
    for i, (d, slots) in enumerate(_hops(case)):
        d, slots = (d, slots) if i == 0 else (d / 2, slots / 2)
        slots = min(slots, d * (2 * _edges(case) / case["nodes"] + 1))
        total += 16 * d + 8 * slots + 4 * (d + slots) + slots / 8 * (32 + 128 * v) + d / 2
    return total


def work(case):
    op, n, e = case["op"], case["nodes"], ESIZE[case["dtype"]]
    nnz = 2 * _edges(case) + n
    if op == "spmm":
        w = case["width"]
        return {"bytes": 2 * (_graph_bytes(case) + 2 * n * w * e), "flops": 2 * 2.0 * nnz * w}
    if op == "build":
        return {"bytes": 8 * (n + 1) + 8 * nnz + 2 * _graph_bytes(case), "flops": 0}
    if op == "sample":
        return {"bytes": _sampling_bytes(case), "flops": 0}
    f, h, c = case["features"], case["hidden"], case["classes"]
    params = e * (2 * f * h + 2 * h * c)
    if op == "infer":                                 # three layers, each a product with the graph and two with weights
        return {"bytes": _graph_bytes(case) + n * (f + c) * e + params + 2 * h * h * e,
                "flops": 4.0 * n * (f * h + h * h + h * c) + 2.0 * nnz * (min(f, h) + h + c)}
    if op == "epoch":
        # per layer: X W for the neighbours and for the node itself, their weight gradients, the second layer's
        # input gradients; three products with the graph (first layer forward, second layer both ways)
        dense = 4 * 2.0 * n * f * h + 6 * 2.0 * n * h * c
        return {"bytes": 2 * _graph_bytes(case) + n * f * e + 6 * params, "flops": dense + 2.0 * nnz * (min(f, h) + 2 * c)}
    hops = _hops(case)
    dims = [f] + [h] * (len(hops) - 1) + [c]
    flops, read = 0.0, 0.0
    for layer, (d, slots) in enumerate(reversed(hops)):
        d, slots = (d, slots) if layer == len(hops) - 1 else (d / 2, slots / 2)
        flops += (4 if layer == 0 else 6) * 2.0 * d * dims[layer] * dims[layer + 1] + 2 * 2.0 * slots * dims[layer]
        if layer == 0:
            read = (d + slots) * f * e
    return {"bytes": _sampling_bytes(case) + read + 6 * (params + (len(hops) - 2) * 2 * h * h * e), "flops": flops}


def tolerance(case):
    if case["op"] in ("build", "sample"):
        return "exact"                                # index work, and values that are copied
    if case["op"] == "spmm":
        # fp32 graphs are multiplied in TF32 (11 significant bits), half-precision results are rounded once
        return {"rel": 4e-3 if case["dtype"] == "bf16" else 1e-3, "max": 4e-2}
    # Training: a last-bit difference that moves an activation across zero switches a whole term of the weight
    # gradients on or off, and Adam's first steps follow the gradients' signs.  Two exact-enough products (TF32
    # against fp32, two summation orders of 16-bit results) leave the gradients of the first steps up to this far
    # apart.
    return {"rel": {"f32": 2e-2, "f16": 2e-2, "bf16": 3e-2}[case["dtype"]], "max": 0.8}
