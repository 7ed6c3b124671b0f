"""What the framework is timed on: one pass of the calls that a user's training or inference program makes.

Five kinds of work, each through the public operators, layers and samplers:

  aggr    neighbourhood aggregation (sum, mean, per-edge values) over a CSR graph, inference or forward + gradient
  gat     a GAT layer, inference or forward + the gradients of its input and parameters
  rgcn    an RGCN layer, inference or forward + gradients
  typed   the per-edge typed linear with its two gradients, relation buckets prepared once per graph
  batch   one mini-batch: sample the neighbourhood of the seeds, gather features, run the model (and its backward)

Graphs follow the power law of `cxgnncomp.synthetic` (symmetrised, one self-loop per node), the shapes those of the
benchmark configurations or fractions of them; features are N(0, 1) like those the models see after normalisation.
"""
import functools
import math
import os
import sys

import numpy as np
import torch
import torch.nn.functional as F

# the working folder is the root of the repository whose code is run
_PKG = os.path.join(os.getcwd(), "cxgnn-compute_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cxgnncomp  # noqa: E402
import cxgnncomp_backend as be  # noqa: E402
from cxgnncomp import synthetic  # noqa: E402

_DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}
_ELEM = {"fp32": 4, "bf16": 2}
_INDEX = {"int64": torch.int64, "int32": torch.int32}


def _aggr(nodes, und, feat, dtype, index, reduce, train):
    return {"kind": "aggr", "nodes": nodes, "undirected": und, "feat": feat, "dtype": dtype, "index": index,
            "reduce": reduce, "train": train}


def _gat(nodes, und, in_feat, heads, channels, concat, train):
    return {"kind": "gat", "nodes": nodes, "undirected": und, "in_feat": in_feat, "heads": heads,
            "channels": channels, "concat": concat, "train": train}


def _rgcn(nodes, und, in_feat, out_feat, rel, dtype, train):
    return {"kind": "rgcn", "nodes": nodes, "undirected": und, "in_feat": in_feat, "out_feat": out_feat, "rel": rel,
            "dtype": dtype, "train": train}


def _typed(edges, in_feat, out_feat, rel, dtype):
    return {"kind": "typed", "edges": edges, "in_feat": in_feat, "out_feat": out_feat, "rel": rel, "dtype": dtype}


def _batch(model, nodes, und, feat, hidden, classes, fanouts, seeds, train):
    return {"kind": "batch", "model": model, "nodes": nodes, "undirected": und, "feat": feat, "hidden": hidden,
            "classes": classes, "fanouts": fanouts, "seeds": seeds, "train": train}


def listed():
    return [
        # the aggregation of one small sub-graph, as a served request or the last layer of a sampled batch has it:
        # what counts is the time of the call itself
        dict(_aggr(1000, 5000, 64, "fp32", "int64", "mean", False), name="aggr_subgraph_infer"),
        # GCN aggregation of configuration 1 with the gradient of the features: the step of full-graph training
        dict(_aggr(169_343, 1_081_572, 128, "fp32", "int64", "sum", True), name="aggr_arxiv_train"),
        # normalised aggregation of class scores (47 classes) with per-edge values, as the last layer of a full-graph
        # GCN has it: rows of an odd width
        dict(_aggr(244_903, 6_185_000, 47, "fp32", "int64", "value", True), name="aggr_classes_train"),
        # first layer of full-graph mean aggregation on the graph of configuration 3 (100 input features): inference
        # over all nodes
        dict(_aggr(2_449_029, 61_850_000, 100, "fp32", "int64", "mean", False), name="aggr_products_infer"),
        # one GPU's eighth of the nodes and edges of configuration 5, bf16 features and 32-bit ids: the largest
        dict(_aggr(13_875_000, 93_062_500, 128, "bf16", "int32", "sum", False), name="aggr_papers_infer"),
        # the GAT layer of configuration 2
        dict(_gat(169_343, 1_081_572, 128, 4, 32, True, True), name="gat_arxiv_train"),
        # the last layer of a GAT stack in inference: heads averaged, one column per class
        dict(_gat(169_343, 1_081_572, 128, 4, 47, False, False), name="gat_classes_infer"),
        # the RGCN layer of configuration 4 in bf16: inference over all nodes
        dict(_rgcn(1_940_000, 9_530_000, 128, 64, 8, "bf16", False), name="rgcn_infer_bf16"),
        # the same layer in fp32 with its gradients, on a quarter of the nodes and edges
        dict(_rgcn(485_000, 2_382_500, 128, 64, 8, "fp32", True), name="rgcn_train_fp32"),
        # per-edge typed linear with both gradients on the edges of configuration 1
        dict(_typed(2_332_487, 128, 64, 8, "fp32"), name="typed_linear_train"),
        # one training step of configuration 3 up to the gradients: sample, gather, forward, backward
        dict(_batch("SAGE", 2_449_029, 61_850_000, 100, 256, 47, "15,10,5", 1024, True), name="sage_batch_train"),
        # the same model answering for a handful of nodes
        dict(_batch("SAGE", 244_903, 6_185_000, 100, 256, 47, "15,10,5", 32, False), name="sage_batch_infer"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["aggr", "gat", "rgcn", "typed", "batch"], [5, 2, 2, 1, 2])[0]
    if kind == "aggr":
        nodes = _log(rng, 700, 6_000_000)
        und = min(int(nodes * math.exp(rng.uniform(math.log(2.0), math.log(26.0)))), 40_000_000)
        # feature widths: half of them the round ones that layers are given, half of them any (class counts, raw
        # features)
        feat = rng.choice([16, 32, 64, 96, 128, 192, 256]) if rng.random() < 0.5 else _log(rng, 8, 256)
        reduce = rng.choice(["sum", "mean", "value"])
        dtype = rng.choice(["fp32", "fp32", "bf16"])
        train = rng.random() < 0.5
        # no more values gathered than in the largest listed case
        und = min(und, int(0.8e10 / ((2 if train else 1) * feat * (2 if dtype == "bf16" else 4) / 2)) - nodes // 2)
        return _aggr(nodes, und, feat, dtype, rng.choice(["int64", "int32"]), reduce, train)
    if kind == "gat":
        nodes = _log(rng, 700, 300_000)
        und = int(nodes * math.exp(rng.uniform(math.log(2.0), math.log(20.0))))
        heads = rng.choice([1, 2, 4, 8])
        train = rng.random() < 0.6
        # the gradients take powers of two
        channels = rng.choice([8, 16, 32, 64]) if train or rng.random() < 0.3 else rng.randint(5, 64)
        in_feat = rng.choice([32, 64, 128, 256]) if train else rng.choice([32, 64, 100, 128, 256])
        return _gat(nodes, und, in_feat, heads, channels, heads > 1 and rng.random() < 0.6, train)
    if kind == "rgcn":
        nodes = _log(rng, 2000, 1_000_000)
        und = int(nodes * math.exp(rng.uniform(math.log(2.0), math.log(10.0))))
        return _rgcn(nodes, und, rng.choice([32, 64, 96, 128]), rng.choice([16, 32, 48, 64, 128]), rng.randint(2, 12),
                     rng.choice(["fp32", "bf16"]), rng.random() < 0.5)
    if kind == "typed":
        return _typed(_log(rng, 3000, 4_000_000), 16 * rng.randint(1, 8), 16 * rng.randint(1, 8), rng.randint(2, 12),
                      rng.choice(["fp32", "bf16"]))
    nodes = _log(rng, 20_000, 1_500_000)
    und = int(nodes * math.exp(rng.uniform(math.log(3.0), math.log(25.0))))
    return _batch(rng.choice(["SAGE", "SAGE", "GIN"]), nodes, und, _log(rng, 32, 300), rng.choice([64, 128, 256]),
                  rng.randint(5, 180), rng.choice(["15,10,5", "10,10", "10,10,10", "25,10", "5,5,5"]),
                  _log(rng, 16, 1024), rng.random() < 0.6)


# ----------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=2)
def _rank_cdf(n):
    """Distribution over the ranks of `synthetic.powerlaw_graph`, summed on the host: always the same bits."""
    cdf = np.cumsum(np.arange(1, n + 1, dtype=np.float64) ** (-1.0 / 1.1))
    return torch.from_numpy(cdf / cdf[-1])


def _graph(case, seed, index=torch.int64):
    """(ptr int64, idx) of the case's graph: the one `synthetic.powerlaw_graph` describes, from the seed alone (its
    own running sum of the weights on the GPU is not the same twice)."""
    n, und = case["nodes"], case["undirected"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    cdf = _rank_cdf(n).cuda()
    perm = torch.randperm(n, generator=gen, device="cuda")

    def ends(k):
        r = torch.rand(k, dtype=torch.float64, device="cuda", generator=gen)
        return perm[torch.searchsorted(cdf, r).clamp_(max=n - 1)]

    u, v = ends(und), ends(und)
    v = torch.where(u == v, (v + 1) % n, v)
    loops = torch.arange(n, device="cuda")
    keys = torch.cat([v * n + u, u * n + v, loops * n + loops])
    del u, v
    keys = torch.sort(keys).values
    ptr = torch.searchsorted(keys, torch.arange(n + 1, dtype=torch.int64, device="cuda") * n)
    return ptr, keys.remainder_(n).to(index)


def _nnz(case):
    return 2 * case["undirected"] + case["nodes"]


def prepare(case, seed):
    kind = case["kind"]
    torch.manual_seed(seed)
    st = {"kind": kind}
    if kind == "aggr":
        dtype = _DTYPES[case["dtype"]]
        st["ptr"], st["idx"] = _graph(case, seed, _INDEX[case["index"]])
        st["n"] = case["nodes"]
        st["x"] = synthetic.node_features(case["nodes"], case["feat"], seed=seed, device="cuda", dtype=dtype)
        st["reduce"] = case["reduce"]
        st["train"] = case["train"]
        if case["reduce"] == "value":  # the 1 / in-degree weights of a normalised GCN
            st["val"] = be.edge_value_degree(st["ptr"], case["nodes"], st["idx"].shape[0])
        if case["train"]:
            st["x"].requires_grad_(True)
            st["g"] = synthetic.node_features(case["nodes"], case["feat"], seed=seed + 1, device="cuda", dtype=dtype)
        return st
    if kind == "gat":
        st["ptr"], st["idx"] = _graph(case, seed)
        st["n"] = case["nodes"]
        st["conv"] = cxgnncomp.MyGATConv(case["in_feat"], case["channels"], heads=case["heads"],
                                         concat=case["concat"]).cuda()
        st["x"] = synthetic.node_features(case["nodes"], case["in_feat"], seed=seed, device="cuda")
        st["train"] = case["train"]
        if not case["train"]:
            return st
        st["x"].requires_grad_(True)
        width = case["heads"] * case["channels"] if case["concat"] else case["channels"]
        st["g"] = synthetic.node_features(case["nodes"], width, seed=seed + 1, device="cuda")
        return st
    if kind == "rgcn":
        dtype = _DTYPES[case["dtype"]]
        st["ptr"], st["idx"] = _graph(case, seed)
        st["n"] = case["nodes"]
        st["rel"] = synthetic.edge_relations(st["idx"].shape[0], case["rel"], seed=seed, device="cuda")
        st["conv"] = cxgnncomp.MyRGCNConv(case["in_feat"], case["out_feat"], case["rel"]).cuda().to(dtype)
        st["x"] = synthetic.node_features(case["nodes"], case["in_feat"], seed=seed, device="cuda", dtype=dtype)
        st["train"] = case["train"]
        if case["train"]:
            st["x"].requires_grad_(True)
            st["g"] = synthetic.node_features(case["nodes"], case["out_feat"], seed=seed + 1, device="cuda", dtype=dtype)
        return st
    if kind == "typed":
        dtype = _DTYPES[case["dtype"]]
        st["types"] = synthetic.edge_relations(case["edges"], case["rel"], seed=seed, device="cuda")
        st["w"] = synthetic.xavier_uniform((case["rel"], case["in_feat"], case["out_feat"]), case["in_feat"],
                                           case["out_feat"], seed=seed, device="cuda", dtype=dtype).requires_grad_(True)
        st["x"] = synthetic.node_features(case["edges"], case["in_feat"], seed=seed, device="cuda",
                                          dtype=dtype).requires_grad_(True)
        st["g"] = synthetic.node_features(case["edges"], case["out_feat"], seed=seed + 1, device="cuda", dtype=dtype)
        st["buckets"] = cxgnncomp.TypedLinearE2EOP.preprocess(st["w"], st["types"])
        return st
    ptr, idx = _graph(case, seed)
    fanouts = [int(f) for f in case["fanouts"].split(",")]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    st["x"] = synthetic.node_features(case["nodes"], case["feat"], seed=seed, device="cuda")
    st["y"] = torch.randint(0, case["classes"], (case["nodes"],), device="cuda", generator=gen)
    st["sampler"] = cxgnncomp.NeighborSampler(ptr, idx, fanouts)
    # no dropout, so that a pass gives the same values whatever was drawn before it
    st["model"] = cxgnncomp.get_model_from_str(case["model"], case["feat"], case["hidden"], case["classes"],
                                               len(fanouts), dropout=0.0).cuda()
    st["params"] = list(st["model"].parameters())
    st["train"] = case["train"]
    if not case["train"]:
        st["model"].eval()
    st["order"] = torch.randperm(case["nodes"], device="cuda", generator=gen)
    st["seeds"] = case["seeds"]
    st["step"] = 0
    return st


def run(st):
    kind = st["kind"]
    if kind == "aggr":
        def forward():
            if st["reduce"] == "sum":
                return be.sage_sum_forward(st["x"], st["ptr"], st["idx"], st["n"])
            if st["reduce"] == "mean":
                return be.sage_mean_forward(st["x"], st["ptr"], st["idx"], st["n"])
            return be.sage_sum_forward_edge_value(st["x"], st["ptr"], st["idx"], st["val"], st["n"])

        if not st["train"]:
            with torch.no_grad():
                return forward()
        y = forward()
        (gx,) = torch.autograd.grad(y, [st["x"]], st["g"])
        return y.detach(), gx
    if kind == "gat":
        conv = st["conv"]
        if not st["train"]:
            with torch.no_grad():
                return conv(st["x"], st["ptr"], st["idx"], st["n"], st["n"], st["idx"].shape[0])
        y = conv(st["x"], st["ptr"], st["idx"], st["n"], st["n"], st["idx"].shape[0])
        grads = torch.autograd.grad(y, [st["x"], conv.lin_src, conv.att_src, conv.att_dst, conv.bias], st["g"])
        return [y.detach(), *grads]
    if kind == "rgcn":
        conv = st["conv"]
        if not st["train"]:
            with torch.no_grad():
                return conv(st["x"], st["ptr"], st["idx"], st["rel"], st["n"])
        y = conv(st["x"], st["ptr"], st["idx"], st["rel"], st["n"])
        grads = torch.autograd.grad(y, [st["x"], conv.linear], st["g"])
        return [y.detach(), *grads]
    if kind == "typed":
        y = cxgnncomp.TypedLinearE2EOP.apply(st["x"], st["w"], st["types"], st["buckets"])
        grads = torch.autograd.grad(y, [st["x"], st["w"]], st["g"])
        return [y.detach(), *grads]
    n = st["order"].shape[0]
    at = st["step"] * st["seeds"] % max(1, n - st["seeds"])
    seeds = st["order"][at:at + st["seeds"]]
    st["step"] += 1
    batch = st["sampler"].batch(st["x"], seeds, seed=st["step"], y=st["y"])
    if not st["train"]:
        with torch.no_grad():
            return st["model"](batch)
    out = st["model"](batch)
    loss = F.nll_loss(out, batch.y)
    grads = torch.autograd.grad(loss, st["params"])
    # one flat gradient, the form in which a data-parallel program reduces it
    return {"out": out.detach(), "loss": loss.detach(), "grad": torch.cat([g.reshape(-1) for g in grads])}


# ----------------------------------------------------------------------------------------------------------------
def _reached(case):
    """Expected distinct nodes after every hop (seeds first) and sampled edges: nodes in classes of like rank, a draw
    reaches a node in proportion to its degree (the law of `synthetic.powerlaw_graph`)."""
    n = case["nodes"]
    rank = np.unique(np.geomspace(1, n + 1, 400).astype(np.int64))
    count = np.diff(rank).astype(np.float64)
    weight = ((rank[:-1] + rank[1:]) / 2.0) ** (-1.0 / 1.1)
    deg = 2.0 * case["undirected"] * weight / (count * weight).sum() + 1.0
    known = count * min(1.0, case["seeds"] / n)
    front, nodes, edges = known, [float(known.sum())], 0.0
    for f in case["fanouts"].split(","):
        picked = float((front * np.minimum(deg, int(f))).sum())
        edges += picked
        front = (count - known) * -np.expm1(-picked * deg / (count * deg).sum())
        known = known + front
        nodes.append(float(known.sum()))
    return nodes, edges


def work(case):
    kind = case["kind"]
    if kind == "aggr":
        n, nnz, f, e = case["nodes"], _nnz(case), case["feat"], _ELEM[case["dtype"]]
        graph = nnz * (8 if case["index"] == "int64" else 4) + (n + 1) * 8
        per_edge = nnz * 4 if case["reduce"] == "value" else 0
        once = 2 * n * f * e + graph + per_edge
        passes = 2 if case["train"] else 1
        return {"bytes": passes * once, "flops": passes * (2 if case["reduce"] == "value" else 1) * nnz * f}
    if kind == "gat":
        n, nnz, k = case["nodes"], _nnz(case), case["in_feat"]
        w = case["heads"] * case["channels"]
        out = w if case["concat"] else case["channels"]
        if not case["train"]:
            # x in, the transformed features out and in, the output out, the graph
            return {"bytes": n * 4 * (k + 2 * w + out) + nnz * 8 + (n + 1) * 8, "flops": 2 * n * k * w + nnz * 2 * w}
        # x in twice, its gradient out, the transformed features out and in for each direction, the output out, its
        # gradient in, the graph once for each direction
        nbytes = n * 4 * (3 * k + 4 * w + 2 * out) + 2 * (nnz * 8 + (n + 1) * 8)
        return {"bytes": nbytes, "flops": 6 * n * k * w + nnz * 8 * w}
    if kind == "rgcn":
        n, nnz, k, o, e = case["nodes"], _nnz(case), case["in_feat"], case["out_feat"], _ELEM[case["dtype"]]
        graph = nnz * 16 + (n + 1) * 8
        weights = case["rel"] * k * o * e
        dense = 2.0 * min(nnz, n * case["rel"]) * k * o
        if case["train"]:
            return {"bytes": n * e * (3 * k + 2 * o) + 2 * graph + 3 * weights, "flops": 3 * dense}
        return {"bytes": n * e * (k + o) + graph + weights, "flops": dense}
    if kind == "typed":
        m, k, o, e = case["edges"], case["in_feat"], case["out_feat"], _ELEM[case["dtype"]]
        return {"bytes": m * e * (3 * k + 3 * o) + 3 * m * 8 + 3 * case["rel"] * k * o * e, "flops": 6.0 * m * k * o}
    nodes, edges = _reached(case)
    fanouts = case["fanouts"].split(",")
    dims = [case["feat"]] + [case["hidden"]] * (len(fanouts) - 1) + [case["classes"]]
    mats = 2 if case["model"] == "SAGE" else 1
    flops, nbytes = 0.0, edges * 16 + nodes[-1] * (4 * case["feat"] + 8)
    for i in range(len(fanouts)):
        rows = nodes[len(fanouts) - 1 - i]
        flops += 2.0 * mats * rows * dims[i] * dims[i + 1]
        nbytes += rows * 4 * dims[i + 1] + mats * 4 * dims[i] * dims[i + 1]
    return {"bytes": nbytes * (3 if case["train"] else 1), "flops": flops * (3 if case["train"] else 1)}


def tolerance(case):
    if case.get("dtype") == "bf16":
        return {"rel": 1e-2, "max": 0.1}
    if case["kind"] == "batch":
        # fp32, but an activation within rounding of zero may fall on either side of the ReLU
        return {"rel": 1e-4, "max": 1e-2}
    return {"rel": 1e-5, "max": 1e-3}
