"""The performance cases of this package: what its users run, over the sizes they run it at.

Everything goes through the public surface -- `QLinear`, the autograd operators of `SPMM` / `SDDMM` and the evaluation
models of `gnn` -- on seeded synthetic inputs.  A training pass is forward + loss + backward (the reference times
exactly that, without the optimizer step, evaluation/test_gcn.py:241-267); its outputs are the results and every
gradient.  Graphs are the seeded R-MAT graphs with one self loop per node that stand in for citation, co-purchase and
social networks: from a few thousand nodes to 232,965 nodes / 114.6 M edges.
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

import tango_b200 as T
from tango_b200 import config, kernels
from tango_b200.gnn import GAT, GCN, HGT
from tango_b200.graph import rmat_graph

MAX_NODES, MAX_EDGES = 232_965, 114_615_892 - 232_965
MID = {"nodes": 169_343, "edges": 1_166_243}
BIG = {"nodes": MAX_NODES, "edges": MAX_EDGES}
SMALL = {"nodes": 19_717, "edges": 88_648}


def listed():
    return [
        # one linear layer of a small model, forward + backward: a few microseconds of work, all launches and host time
        {"name": "qlinear_small", "kind": "qlinear", "m": 2000, "k": 100, "n": 32, "bias": True, "rounding": "reference"},
        # the input layer of a full-graph model: long, ragged rows (602 features are 2408 bytes)
        {"name": "qlinear_large", "kind": "qlinear", "m": 232_965, "k": 602, "n": 256, "bias": True,
         "rounding": "reference"},
        # a wide hidden layer: the most arithmetic per byte that graph models bring
        {"name": "qlinear_wide", "kind": "qlinear", "m": 131_072, "k": 1024, "n": 1024, "bias": False,
         "rounding": "nearest"},
        # neighbour sum as an operator, both directions, on a sparse graph (8 edges per node)
        {"name": "spmm_mid", "kind": "spmm", **MID, "f": 128, "rounding": "reference"},
        # multi-head edge scores as an operator, both directions
        {"name": "edge_dot_mid", "kind": "edge_dot", **MID, "heads": 4, "d": 32, "rounding": "reference"},
        # training epoch of a small citation network: launch latency and host time
        {"name": "gcn_small", "kind": "gcn", **SMALL, "feats": 500, "hidden": 16, "classes": 3, "layers": 1, "train": True,
         "rounding": "reference"},
        # three layers on a sparse graph with stochastic rounding (hidden layers aggregate before they multiply)
        {"name": "gcn_mid", "kind": "gcn", **MID, "feats": 128, "hidden": 128, "classes": 40, "layers": 2, "train": True,
         "rounding": "stochastic"},
        # training epoch of the full-graph benchmark
        {"name": "gcn_large", "kind": "gcn", **BIG, "feats": 602, "hidden": 256, "classes": 41, "layers": 1, "train": True,
         "rounding": "reference"},
        # evaluation pass (forward only) between training epochs, on a graph of 86 edges per node
        {"name": "gcn_eval", "kind": "gcn", "nodes": 232_965, "edges": 20_000_000, "feats": 602, "hidden": 256,
         "classes": 41, "layers": 1, "train": False, "rounding": "reference"},
        # attention model on the small citation network: eight narrow heads
        {"name": "gat_small", "kind": "gat", **SMALL, "feats": 500, "hidden": 8, "classes": 3, "heads": 8,
         "attention": "fp32", "rounding": "reference"},
        # attention model on the full graph
        {"name": "gat_large", "kind": "gat", **BIG, "feats": 602, "hidden": 64, "classes": 41, "heads": 4,
         "attention": "fp32", "rounding": "reference"},
        # graph-transformer layer: six projections, dot-product attention
        {"name": "hgt_mid", "kind": "hgt", **MID, "feats": 128, "out": 128, "heads": 4, "rounding": "reference"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _graph_size(rng, max_edges):
    """A node count and an edge count: 4 edges per node up to the density of the full-graph benchmark (n^1.5 edges)."""
    n = _log(rng, 2000, MAX_NODES)
    return {"nodes": n, "edges": _log(rng, 4 * n, min(max_edges, max(8 * n, int(n ** 1.5 * 0.9))))}


def draw(rng):
    kind = rng.choice(["qlinear", "qlinear", "spmm", "edge_dot", "gcn", "gcn", "gat", "hgt"])
    c = {"kind": kind, "rounding": rng.choice(["reference", "reference", "nearest", "stochastic"])}
    if kind == "qlinear":
        c.update(m=_log(rng, 1000, 232_965), k=_log(rng, 16, 1024), n=_log(rng, 3, 1024), bias=rng.random() < 0.5)
    elif kind == "spmm":
        c.update(_graph_size(rng, 20_000_000), f=_log(rng, 3, 602))
    elif kind == "edge_dot":
        c.update(_graph_size(rng, 12_000_000), heads=rng.choice([1, 1, 2, 4, 8]), d=8 * _log(rng, 1, 8))
        if c["heads"] == 1:
            c["d"] = _log(rng, 8, 256)
    elif kind == "gcn":
        c.update(_graph_size(rng, MAX_EDGES), feats=_log(rng, 32, 602), hidden=_log(rng, 8, 256), classes=rng.randint(3, 48),
                 layers=rng.choice([1, 1, 2]), train=rng.random() < 0.75)
    elif kind == "gat":
        c.update(_graph_size(rng, 12_000_000), feats=_log(rng, 32, 602), hidden=8 * _log(rng, 1, 8),
                 classes=rng.randint(3, 48), heads=rng.choice([1, 2, 4, 4, 8]), attention=rng.choice(["fp32", "fp32", "int8"]))
        c["hidden"] = min(c["hidden"], 256 // c["heads"])
    else:
        heads = rng.choice([1, 2, 4, 8])
        c.update(_graph_size(rng, 12_000_000), feats=_log(rng, 32, 602), heads=heads, out=heads * 8 * _log(rng, 1, 32 // heads))
    return c


def _graph(case, seed):
    return T.graph_preprocess(rmat_graph(case["nodes"], case["edges"], seed, device="cuda"))


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    torch.cuda.manual_seed(seed)

    def randn(*shape):
        return torch.randn(shape, device="cuda", generator=gen)

    kind = case["kind"]
    s = {"kind": kind, "rounding": case["rounding"], "seed": seed}
    if kind == "qlinear":
        s["layer"] = T.QLinear(case["k"], case["n"], bias=case["bias"]).cuda()
        s["x"] = randn(case["m"], case["k"]).requires_grad_()
        s["grad"] = randn(case["m"], case["n"]) / case["m"]
        return s
    g = s["graph"] = _graph(case, seed)
    n = case["nodes"]
    if kind == "spmm":
        s["x"] = randn(n, case["f"]).requires_grad_()
        s["grad"] = randn(n, case["f"]) / n
    elif kind == "edge_dot":
        s["u"] = randn(n, case["heads"], case["d"]).requires_grad_()
        s["v"] = randn(n, case["heads"], case["d"]).requires_grad_()
        s["grad"] = randn(g.num_edges(), case["heads"], 1) / n
    else:
        s["x"] = randn(n, case["feats"])
        if kind == "gcn":
            s["model"] = GCN(g, case["feats"], case["hidden"], case["classes"], case["layers"]).cuda()
            s["train"] = case["train"]
        elif kind == "gat":
            fused = "int8" if case["attention"] == "int8" else True
            s["model"] = GAT(g, 2, case["feats"], case["hidden"], case["classes"], [case["heads"], 1], fused=fused).cuda()
        else:
            s["model"] = HGT(case["feats"], case["out"], case["heads"]).cuda()
            s["grad"] = randn(n, case["out"]) / n
        if kind in ("gcn", "gat"):
            s["labels"] = torch.randint(0, case["classes"], (n,), device="cuda", generator=gen)
    return s


def run(s):
    config.set_rounding(s["rounding"], s["seed"])
    kernels.set_call_counter(0)     # stochastic rounding draws the same numbers in every pass
    kind = s["kind"]
    if kind == "qlinear":
        layer, x = s["layer"], s["x"]
        layer.zero_grad(set_to_none=True)
        x.grad = None
        y = layer(x)
        y.backward(s["grad"])
        return [y.detach(), x.grad] + [p.grad for p in layer.parameters()]
    if kind == "spmm":
        x = s["x"]
        x.grad = None
        out = T.spmm_copy_u.apply(s["graph"], x)
        out.backward(s["grad"])
        return out.detach(), x.grad
    if kind == "edge_dot":
        u, v = s["u"], s["v"]
        u.grad = v.grad = None
        out = T.sddmm_u_dot_v.apply(s["graph"], u, v)
        out.backward(s["grad"])
        return out.detach(), u.grad, v.grad
    model = s["model"]
    if kind == "gcn" and not s["train"]:
        with torch.no_grad():
            return model(s["x"])
    model.zero_grad(set_to_none=True)
    if kind == "hgt":
        out = model(s["graph"], s["x"])
        out.backward(s["grad"])
        return [out.detach()] + [p.grad for p in model.parameters()]
    logits = model(s["x"])
    loss = F.cross_entropy(logits, s["labels"])
    loss.backward()
    return [loss.detach(), logits.detach()] + [p.grad for p in model.parameters()]


def work(case):
    """Every input and output once, in fp32; every edge's index once per direction of the graph that the pass walks."""
    kind = case["kind"]
    if kind == "qlinear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4 * (2 * m * k + 2 * m * n + 2 * n * k + 2 * n * case["bias"]), "flops": 6 * m * n * k}
    n, e = case["nodes"], case["edges"] + case["nodes"]
    both = 8 * (e + n)                                             # CSC and CSR: indptr and indices
    if kind == "spmm":
        return {"bytes": both + 16 * n * case["f"], "flops": 2 * e * case["f"]}
    if kind == "edge_dot":
        f, h = case["heads"] * case["d"], case["heads"]
        return {"bytes": both + 16 * n * f + 8 * e * h, "flops": 6 * e * f}
    if kind == "gcn":
        widths = [case["feats"]] + [case["hidden"]] * case["layers"] + [case["classes"]]
        flops = 0
        for i, (a, b) in enumerate(zip(widths, widths[1:])):
            gemm, agg = 2 * n * a * b, e * min(a, b)
            flops += gemm + agg
            if case["train"]:
                flops += gemm * (2 if i else 1) + agg              # dW everywhere, dX below the first layer
        params = sum(a * b + b for a, b in zip(widths, widths[1:]))
        nbytes = 4 * n * (widths[0] + widths[-1]) + 4 * params * (2 if case["train"] else 1)
        return {"bytes": nbytes + (both + 8 * n if case["train"] else both // 2), "flops": flops}
    if kind == "gat":
        wide = case["heads"] * case["hidden"]
        flops = 4 * n * case["feats"] * wide + 6 * n * wide * case["classes"]
        flops += 6 * e * (wide + case["classes"]) + 20 * e * (case["heads"] + 1)   # aggregation, its two gradients, softmax
        params = case["feats"] * wide + wide * case["classes"] + 3 * (wide + case["classes"])
        return {"bytes": both + 8 * n + 4 * n * (case["feats"] + case["classes"]) + 8 * params, "flops": flops}
    f, o = case["feats"], case["out"]
    flops = 3 * 4 * n * f * o + 3 * 6 * n * o * o + 12 * e * o + 20 * e * case["heads"]
    return {"bytes": both + 4 * n * (f + 2 * o) + 8 * (3 * f * o + 3 * o * o + 6 * o), "flops": flops}


def tolerance(case):
    """Single operators: exact int32 sums of int8 codes, scaled in fp32; an absmax scale that is one ulp off moves about one
    code in 10^5 to its neighbour, which is 1e-4 of a result.  Models chain up to a dozen of them, and every
    requantisation (steps of 1/127 of the largest value) passes such a step on: 1e-2, as for 8 bits of mantissa."""
    return {"rel": 1e-4} if case["kind"] in ("qlinear", "spmm", "edge_dot") else {"rel": 1e-2}
