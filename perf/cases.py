"""Timed cases of the framework: the calls a user's program makes, over the sizes it makes them at.

Six kinds of work, each through the package's public entry points:

  attention   ``sparse_graph_attention`` on a prebuilt ``SparseGraph``, forward and backward or forward alone
  layout      ``SparseGraph`` from an uploaded edge list, both orientations
  batch       ``get_batch_reorder_blockize`` on the whole graph, then the batch's ``SparseGraph``
  evaluate    node-level ``Graphormer`` in evaluation mode
  train       node-level ``Graphormer``, forward, loss and backward into the ``Reducer``'s flat gradients
  graphs      graph-level ``GTGraphLevel`` on a batch of padded graphs, from the raw edge lists to the gradients

Edge lists follow ``torchgt_b200.synthetic.clustered_edges`` (self loops, a global token at row 0 linked both ways
with every node, random edges that mostly stay inside one of eight clusters, optionally power-law sources), made on
the GPU.  Dropout is off in the models: its masks would hide what is compared.
"""
from __future__ import annotations

import math
import random
from types import SimpleNamespace

import torch
from torch.nn import functional as F

from torchgt_b200 import SparseGraph, prepare_edges, sparse_graph_attention
from torchgt_b200.gt import GTGraphLevel
from torchgt_b200.gt_sp.batching import get_batch_reorder_blockize
from torchgt_b200.gt_sp.reducer import Reducer
from torchgt_b200.graphormer import Graphormer

CLUSTERS = 8
GRAPHS = 16          # graphs per batch of the graph-level model
NODE_FEATURES = 5    # integer features per node of the graph-level model
LAYERS, HEADS, HIDDEN = 4, 8, 64


def _attention(name, nodes, random_edges, heads=8, head_dim=8, dtype="fp32", bias="none", backward=True, zipf=0.0):
    case = {"kind": "attention", "nodes": nodes, "random_edges": random_edges, "heads": heads, "head_dim": head_dim,
            "dtype": dtype, "bias": bias, "backward": backward, "zipf": zipf}
    return dict(case, name=name) if name else case


def _graphormer(name, kind, nodes, random_edges, features, classes, tf32):
    case = {"kind": kind, "nodes": nodes, "random_edges": random_edges, "features": features, "classes": classes,
            "tf32": tf32}
    return dict(case, name=name) if name else case


def _batch(name, total_nodes, total_edges, seq_len, batch_nodes, reorder, block_size):
    case = {"kind": "batch", "total_nodes": total_nodes, "total_edges": total_edges, "seq_len": seq_len,
            "batch_nodes": batch_nodes, "reorder": reorder, "block_size": block_size, "features": 128}
    return dict(case, name=name) if name else case


def listed():
    return [
        # one layer's attention in a training step on a small batch: latency, launches and host work
        _attention("attention-4k", 4096, 8 * 4096),
        # the same at sequence length 64,000 with a learnt scalar bias per edge: the benchmark batch
        _attention("attention-64k-dbias", 64000, 334450, bias="edge-grad"),
        # 64,000 nodes in bf16, the form the models use (no bias)
        _attention("attention-64k-bf16", 64000, 334450, dtype="bf16"),
        # the long-sequence batch: 870,000 nodes, 18.2 M edges, power-law sources; K and V exceed the L2
        _attention("attention-870k", 870000, 18214272 - 3 * 870000, zipf=2.1),
        # evaluation: forward alone on the epoch's shorter last batch, 4 heads x 16
        _attention("attention-37k-forward", 37608, 228357 - 3 * 37608, heads=4, head_dim=16, backward=False),
        # what one of eight sequence-parallel ranks computes: all rows of 8 x 64,000, one head of 8
        _attention("attention-512k-1head", 512000, 8 * 334450, heads=1),
        # set-up of the long-sequence batch: both segment layouts from the int64 list as it was uploaded
        {"name": "layout-870k", "kind": "layout", "nodes": 870000, "random_edges": 18214272 - 3 * 870000, "zipf": 2.1,
         "int32": False},
        # a training batch of 64,000 random nodes cut from a graph of 169,343 nodes and 1.17 M edges
        _batch("batch-64k", 169343, 1166243, 64000, 64000, False, 16),
        # the epoch's shorter last batch, its edges regrouped into cluster-sparse blocks
        _batch("batch-37k-blocks", 169343, 1166243, 64000, 37608, True, 16),
        # serving a small graph: the model's forward, bound by launches and host work; fp32 products
        _graphormer("evaluate-4k", "evaluate", 4096, 8 * 4096, 128, 40, False),
        # a training iteration at sequence length 64,000, library products in TF32 as the benchmark sets them
        _graphormer("train-64k", "train", 64000, 334450, 128, 40, True),
        # a graph-level training iteration: 16 call graphs of 2,000 to 20,000 nodes, about 2.5 edges per node
        {"name": "graphs-16x20k", "kind": "graphs", "min_nodes": 2000, "max_nodes": 20000, "degree": 2.5, "tf32": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attention"] * 5 + ["layout", "batch", "evaluate", "train", "graphs"])
    nodes = _log_int(rng, 1000, 870000)
    degree = math.exp(rng.uniform(math.log(1.0), math.log(17.0)))
    if kind == "attention":
        heads, head_dim = rng.choice([(8, 8), (8, 8), (8, 8), (4, 16), (8, 16), (16, 8), (4, 8), (2, 8), (1, 8), (12, 8), (2, 32)])
        nodes = min(nodes, 870000 * 64 // max(64, heads * head_dim))
        bias = rng.choice(["none", "none", "edge", "edge-grad", "head-grad"])
        if bias == "head-grad":
            nodes = min(nodes, 200000)
        return _attention(None, nodes, int(nodes * degree), heads, head_dim, rng.choice(["fp32", "fp32", "bf16"]), bias,
                          rng.random() < 0.75, rng.choice([0.0, 2.1]))
    if kind == "layout":
        return {"kind": kind, "nodes": nodes, "random_edges": int(nodes * degree), "zipf": rng.choice([0.0, 2.1]),
                "int32": rng.random() < 0.3}
    if kind == "batch":
        total = _log_int(rng, 20000, 400000)
        seq_len = _log_int(rng, 4000, total // 2)
        last = rng.random() < 0.3
        return _batch(None, total, int(total * rng.uniform(4.0, 12.0)), seq_len,
                      int(seq_len * rng.uniform(0.3, 0.95)) if last else seq_len, rng.random() < 0.4, rng.choice([8, 16]))
    if kind == "graphs":
        largest = _log_int(rng, 3000, 20000)
        return {"kind": kind, "min_nodes": max(500, largest // 10), "max_nodes": largest, "degree": rng.uniform(1.5, 4.0),
                "tf32": rng.random() < 0.5}
    nodes = _log_int(rng, 1000, 170000)
    features, classes = rng.choice([(128, 40), (128, 40), (100, 47)])
    return _graphormer(None, kind, nodes, int(nodes * min(degree, 8.0)), features, classes, rng.random() < 0.5)


# ---- inputs ----------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _zipf_ranks(count, nodes, exponent, gen):
    """Inverse-CDF draws of p(rank) ~ rank^(-1 / (exponent - 1)), ranks 0 .. nodes - 1."""
    alpha = 1.0 / (exponent - 1.0)
    u = torch.rand(count, generator=gen, device="cuda", dtype=torch.float64)
    ranks = (u * (float(nodes) ** (1.0 - alpha) - 1.0) + 1.0) ** (1.0 / (1.0 - alpha)) - 1.0
    return ranks.clamp_(0, nodes - 1).long()


def _edges(case, gen):
    """[2, 3 nodes + random_edges] int64 over rows 0 .. nodes, in no particular order."""
    n, m = case["nodes"], case["random_edges"]
    size = max(1, n // CLUSTERS)
    nodes = torch.arange(1, n + 1, device="cuda")
    zeros = torch.zeros_like(nodes)
    if case.get("zipf", 0.0) > 1.0:
        src = torch.randperm(n, generator=gen, device="cuda")[_zipf_ranks(m, n, case["zipf"], gen)]
    else:
        src = torch.randint(0, n, (m,), generator=gen, device="cuda")
    cross = torch.rand(m, generator=gen, device="cuda") < 0.315
    near = ((src // size) * size + torch.randint(0, size, (m,), generator=gen, device="cuda")).clamp_(max=n - 1)
    dst = torch.where(cross, torch.randint(0, n, (m,), generator=gen, device="cuda"), near)
    return torch.cat([torch.stack([nodes, nodes]), torch.stack([nodes, zeros]), torch.stack([zeros, nodes]),
                      torch.stack([src + 1, dst + 1])], dim=1)


def _edge_count(case):
    return 3 * case["nodes"] + case["random_edges"]


def _graph(case, gen):
    graph = SparseGraph(_edges(case, gen), case["nodes"] + 1)
    if case["kind"] != "evaluate" and case.get("backward", True):
        graph.by_src     # a training program's graph has both orientations from its first step on
    return graph


def _graph_sizes(case):
    """Nodes of every graph of a graph-level batch: part of the case, not of the seed."""
    rng = random.Random(GRAPHS * case["max_nodes"] + case["min_nodes"])
    sizes = [_log_int(rng, case["min_nodes"], case["max_nodes"]) for _ in range(GRAPHS - 1)]
    return sizes + [case["max_nodes"]]


def _graph_edge_counts(case):
    return [int(n * case["degree"]) for n in _graph_sizes(case)]


def _prepare_attention(case, gen):
    dtype = {"fp32": torch.float32, "bf16": torch.bfloat16}[case["dtype"]]
    shape = (case["nodes"] + 1, case["heads"], case["head_dim"])
    q, k, v, dout = (torch.randn(shape, generator=gen, device="cuda").to(dtype) for _ in range(4))
    bias = None
    if case["bias"] != "none":
        columns = (case["heads"],) if case["bias"] == "head-grad" else ()
        bias = torch.randn((_edge_count(case),) + columns, generator=gen, device="cuda") * 0.1
    if case["backward"]:
        for t in (q, k, v):
            t.requires_grad_()
        if case["bias"].endswith("-grad"):
            bias.requires_grad_()
    return SimpleNamespace(q=q, k=k, v=v, dout=dout, bias=bias, graph=_graph(case, gen))


def _below(bound, power, gen):
    """Random whole numbers in [0, bound), element by element, crowded towards 0 by ``power``."""
    u = torch.rand(bound.shape, generator=gen, device="cuda", dtype=torch.float64)
    return torch.minimum((u ** power * bound).long(), bound - 1)


def _prepare_batch(case, gen):
    """How many edges lie inside the batch and which of its clusters they join is part of the case (it sets the
    shape of the result); the rest comes from the seed.  A few nodes have most of the out-edges."""
    n, m, b = case["total_nodes"], case["total_edges"], case["batch_nodes"]
    x = torch.randn(n, case["features"], generator=gen, device="cuda")
    y = torch.randint(0, 40, (n,), generator=gen, device="cuda")
    order = torch.randperm(n, generator=gen, device="cuda")
    idx, others = order[:b], order[b:]
    inside = int(m * (b / n) ** 2)
    fixed = _generator(inside)
    ca = torch.randint(0, CLUSTERS, (inside,), generator=fixed, device="cuda")
    cb = torch.where(torch.rand(inside, generator=fixed, device="cuda") < 0.315,
                     torch.randint(0, CLUSTERS, (inside,), generator=fixed, device="cuda"), ca)
    first = (torch.arange(CLUSTERS + 1, device="cuda") * (b + 1) + CLUSTERS - 1) // CLUSTERS   # of every cluster
    first[0] = 1                                                                               # 0: the global token
    size = first[1:] - first[:-1]
    s, d = _below(size[ca], 3, gen), _below(size[cb], 1, gen)
    d = torch.where((ca == cb) & (s == d), (d + 1) % size[cb], d)                              # no self loops
    within = torch.stack([idx[first[ca] + s - 1], idx[first[cb] + d - 1]])
    rest = torch.full((m - inside,), n, device="cuda")
    leaving = torch.stack([order[_below(rest, 3, gen)], others[_below(rest - b, 1, gen)]])
    edges = torch.cat([within, leaving], dim=1)[:, torch.randperm(m, generator=gen, device="cuda")].contiguous()
    args = SimpleNamespace(seq_len=case["seq_len"], model="graphormer", reorder=case["reorder"])
    return SimpleNamespace(args=args, x=x, y=y, idx=idx, edges=edges)


def _prepare_graphormer(case, gen, seed):
    torch.manual_seed(seed)
    n = case["nodes"]
    model = Graphormer(LAYERS, HEADS, case["features"], HIDDEN, case["classes"], 1, 0.0, 0.0, 0.0, HIDDEN, 1).cuda()
    state = SimpleNamespace(model=model, x=torch.randn(n, case["features"], generator=gen, device="cuda"),
                            graph=_graph(case, gen))
    if case["kind"] == "train":
        model.train()
        state.y = torch.randint(0, case["classes"], (n,), generator=gen, device="cuda")
        state.reducer = Reducer().init(model)
    else:
        model.eval()
    return state


def _prepare_graphs(case, gen, seed):
    torch.manual_seed(seed)
    sizes, counts = _graph_sizes(case), _graph_edge_counts(case)
    raw = []
    for n, m in zip(sizes, counts):      # call graphs: a node is called by earlier ones
        dst = torch.randint(1, n, (m,), generator=gen, device="cuda")
        src = (torch.rand(m, generator=gen, device="cuda") * dst).long()
        raw.append(torch.stack([src, dst]))
    x = torch.randint(1, 7000, (GRAPHS, case["max_nodes"], NODE_FEATURES), generator=gen, device="cuda")
    y = torch.randint(0, 5, (GRAPHS,), generator=gen, device="cuda")
    model = GTGraphLevel(LAYERS, HEADS, HIDDEN, 0.0, 0.0, HIDDEN, "other", "multi_hop", 5, 0.0, 5).cuda().train()
    return SimpleNamespace(model=model, reducer=Reducer().init(model), x=x, y=y, raw=torch.cat(raw, dim=1), sizes=sizes,
                           counts=counts)


def prepare(case, seed):
    gen = _generator(seed)
    kind = case["kind"]
    if "tf32" in case:
        torch.backends.cuda.matmul.allow_tf32 = case["tf32"]
    if kind == "attention":
        state = _prepare_attention(case, gen)
    elif kind == "layout":
        edges = _edges(case, gen)
        state = SimpleNamespace(edges=edges.to(torch.int32) if case["int32"] else edges)
    elif kind == "batch":
        state = _prepare_batch(case, gen)
    elif kind == "graphs":
        state = _prepare_graphs(case, gen, seed)
    else:
        state = _prepare_graphormer(case, gen, seed)
    state.case = case
    return state


# ---- one pass --------------------------------------------------------------------------------------------
def _layout_arrays(graph):
    return [getattr(layout, name) for layout in (graph.by_dst, graph.by_src) for name in ("ptr", "other", "perm", "seg")]


def _run_attention(s):
    if not s.case["backward"]:
        with torch.no_grad():
            return sparse_graph_attention(s.q, s.k, s.v, s.graph, s.bias)
    out = sparse_graph_attention(s.q, s.k, s.v, s.graph, s.bias)
    inputs = [s.q, s.k, s.v] + ([s.bias] if s.bias is not None and s.bias.requires_grad else [])
    return [out.detach(), *torch.autograd.grad(out, inputs, s.dout)]


def _run_batch(s):
    case = s.case
    x, y, edges, _ = get_batch_reorder_blockize(s.args, s.x, s.y, s.idx, [case["batch_nodes"]], s.x.device, s.edges,
                                                case["total_nodes"], CLUSTERS, case["block_size"])
    return [x, y, edges, *_layout_arrays(SparseGraph(edges, case["batch_nodes"] + 1))]


def _run_train(s, output, loss):
    loss.backward()
    s.reducer.synchronize()
    return [loss.detach(), output.detach(), s.reducer.flat_gradients]


def run(state):
    kind = state.case["kind"]
    if kind == "attention":
        return _run_attention(state)
    if kind == "layout":
        return _layout_arrays(SparseGraph(state.edges, state.case["nodes"] + 1))
    if kind == "batch":
        return _run_batch(state)
    if kind == "evaluate":
        with torch.no_grad():
            return state.model(state.x, None, state.graph, attn_type="sparse")
    state.reducer.prepare()
    if kind == "train":
        out = state.model(state.x, None, state.graph, attn_type="sparse")
        return _run_train(state, out, F.nll_loss(out, state.y))
    edges = prepare_edges(state.raw, state.sizes, state.counts, add_global_token=False,
                          rows_per_graph=state.case["max_nodes"])
    graph = SparseGraph(edges, GRAPHS * state.case["max_nodes"])
    out = state.model(SimpleNamespace(x=state.x, edge_index=graph), attn_type="sparse")
    return _run_train(state, out, F.cross_entropy(out, state.y))


# ---- what a pass cannot do without -------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "batch":
        n, m, b = case["total_nodes"], case["total_edges"], case["batch_nodes"]
        share = b / n
        edges = m * share * share + 3 * b        # edges inside the batch, self loops, the global token's edges
        return {"bytes": 16 * m + 8 * b + b * (8 * case["features"] + 16) + 16 * edges + 2 * (12 * edges + 4 * b),
                "flops": 0}
    if kind == "layout":
        e = _edge_count(case)
        return {"bytes": (8 if case["int32"] else 16) * e + 2 * (12 * e + 4 * (case["nodes"] + 2)), "flops": 0}
    if kind == "attention":
        e, elems = _edge_count(case), case["heads"] * case["head_dim"]
        row = (case["nodes"] + 1) * elems * (4 if case["dtype"] == "fp32" else 2)
        values = {"none": 0, "edge": 1, "edge-grad": 1, "head-grad": case["heads"]}[case["bias"]]
        tensors, passes = (8, 2) if case["backward"] else (4, 1)
        copies = 2 if case["backward"] and case["bias"].endswith("-grad") else 1
        return {"bytes": tensors * row + passes * e * (4 if case["bias"] == "none" else 8) + 4 * e * values * copies,
                "flops": e * elems * (14 if case["backward"] else 4)}
    if kind == "graphs":
        rows, e = GRAPHS * case["max_nodes"], sum(_graph_edge_counts(case))
        table = 7000 * HIDDEN
        per_row = LAYERS * 8 * HIDDEN * HIDDEN
        return {"bytes": 8 * NODE_FEATURES * rows + 16 * e + 8 * table + 8 * per_row,
                "flops": 3 * 2 * rows * per_row + LAYERS * e * HIDDEN * 14}
    n, e = case["nodes"], _edge_count(case)
    per_row = case["features"] * HIDDEN + LAYERS * 6 * HIDDEN * HIDDEN + HIDDEN * case["classes"]
    train = kind == "train"
    return {"bytes": 4 * n * (case["features"] + case["classes"]) + 4 * e * (2 if train else 1) + 4 * per_row * (2 if train else 1),
            "flops": (3 if train else 1) * 2 * n * per_row + LAYERS * e * HIDDEN * (14 if train else 4)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("layout", "batch"):
        return "exact"                   # whole numbers, and feature rows copied as they are
    if kind == "attention":
        return {"rel": 1e-5} if case["dtype"] == "fp32" else {"rel": 1e-2}
    # whole models: 32-bit sums through four layers and back; TF32 products carry 11 bits
    return {"rel": 3e-3} if case["tf32"] else {"rel": 2e-5}
