"""The work a user has this framework do, as cases that can be timed and whose outputs can be compared.

A user scores a stream of timed edges with a temporal graph model.  Once per data set the edges become a
time-sorted adjacency on the GPU (``get_neighbor_finder``) and an offline plan says which historical embeddings
to keep after each batch (``get_cache_plan``).  Then the edges are scored batch by batch: one call per batch
(``TGN.compute_edge_probabilities``, or ``TGN.compute_temporal_embeddings`` when the embeddings themselves are
wanted), a whole stream of batches in one call (``TGN.eval_epoch``), or the evaluation loop with its metrics
(``eval_edge_prediction``).  ``NeighborFinder.get_temporal_neighbor`` is called on its own for tables of
neighbours.  Inputs are host arrays wherever the interface takes host arrays.

Sizes are those of the five synthetic workloads in ``orca_b200/synthetic.py`` (the graph families "small" = c1,
"items" = c2 / c3, "nodes" = c4, "large" = c5), and ranges around them.
"""
import argparse
import math
import types

import numpy as np
import torch

from orca_b200 import params
from orca_b200.cache import get_cache_plan
from orca_b200.evaluation import RandEdgeSampler, eval_edge_prediction
from orca_b200.neighbor_finder import get_neighbor_finder
from orca_b200.tgn import TGN

D = 172            # node, edge-feature, time and memory width
ROW = 4 * D        # bytes of one table row
WARM = 2           # batches a prepared model has already scored when the timed ones start


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    small = dict(n_src=1000, n_dst=500, n_edges=20000, zipf_src=1.1, zipf_dst=1.1, times="uniform", span=1e5)
    items = dict(n_src=8227, n_dst=1000, n_edges=157474, zipf_src=1.2, zipf_dst=1.5, times="exp", span=2.7e6)
    items20 = dict(n_src=10000, n_dst=984, n_edges=672447, zipf_src=1.3, zipf_dst=1.3, times="exp", span=2.7e6)
    nodes = dict(n_src=194085, n_dst=0, n_edges=1443339, zipf_src=1.5, zipf_dst=1.5, times="bursty", span=2.3e8)
    large = dict(n_src=1140149, n_dst=0, n_edges=7833140, zipf_src=1.6, zipf_dst=0.0, times="exp", span=2.0e8)
    return [
        # a service that scores a handful of edges as they arrive: one short call, one-layer model
        dict(small, name="call_tiny", kind="score", layers=1, k=10, bs=37, budget=1000, strategy="MRD"),
        # the reference's evaluation loop at its default batch size, one call per batch
        dict(items, name="call_small", kind="score", layers=2, k=10, bs=200, budget=1000, strategy="MRD"),
        # a downstream task takes the embeddings of a large batch on the largest graph
        dict(large, name="call_large", kind="embed", layers=2, k=10, bs=2000, budget=10000, strategy="MRD"),
        # offline scoring of a stretch of the stream in one call: twenty neighbours, LRU plan, short last batch
        dict(items20, name="stream_k20", kind="stream", layers=2, k=20, bs=600, budget=2000, strategy="LRU",
             edges=30311),
        # the same on a graph of users only with a 2Q plan
        dict(nodes, name="stream_nodes", kind="stream", layers=2, k=10, bs=1000, budget=1000, strategy="2Q",
             edges=48000),
        # the headline workload: 2000 edges a batch, 1.14 M nodes, MRD plan
        dict(large, name="stream_large", kind="stream", layers=2, k=10, bs=2000, budget=10000, strategy="MRD",
             edges=100000),
        # exact embeddings: both layers recomputed for every neighbour, no historical embeddings used
        dict(items, name="stream_exact", kind="stream_exact", layers=2, k=10, bs=200, budget=1000, strategy="MRD",
             edges=6100),
        # validation after an epoch: scores and the metrics of every batch
        dict(items, name="evaluate", kind="evaluate", layers=2, k=10, bs=200, budget=1000, strategy="MRD",
             edges=8000),
        # the plan of a stretch of the largest stream
        dict(large, name="plan_mrd", kind="plan", k=10, bs=2000, budget=10000, strategy="MRD", edges=400000),
        # the plan of a smaller stream under LRU, whose evictions are random
        dict(items20, name="plan_lru", kind="plan", k=20, bs=600, budget=2000, strategy="LRU", edges=150000),
        # the adjacency of the largest graph from its edge stream
        dict(large, name="adjacency", kind="adjacency"),
        # the neighbours of every edge's endpoints, as host tables
        dict(items, name="neighbors", kind="neighbors", k=10, queries=39999),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.5:      # users and items
        c = dict(n_src=_log(rng, 500, 12000), n_dst=_log(rng, 100, 1200), n_edges=_log(rng, 20000, 700000),
                 zipf_src=round(rng.uniform(1.1, 1.3), 2), zipf_dst=round(rng.uniform(1.1, 1.5), 2))
    else:                       # users only; on the larger half destinations follow preferential attachment
        c = dict(n_src=_log(rng, 2000, 1140149), n_dst=0, n_edges=_log(rng, 40000, 7833140),
                 zipf_src=round(rng.uniform(1.3, 1.6), 2), zipf_dst=rng.choice([0.0, 1.5]))
    c["times"] = rng.choice(["uniform", "exp", "bursty"])
    c["span"] = float(_log(rng, 1e5, 2.3e8))
    c["kind"] = rng.choice(["score", "score", "embed", "stream", "stream", "stream", "stream_exact", "evaluate", "plan",
                            "adjacency", "neighbors"])
    if c["kind"] == "adjacency":
        return c
    c["k"] = rng.choice([5, 10, 10, 20])
    room = c["n_edges"] // 2     # edges the timed stretch may take (it sits in the second half of the stream)
    if c["kind"] == "neighbors":
        return dict(c, queries=_log(rng, 100, min(200000, 2 * c["n_edges"])))
    most = {"score": 4000, "embed": 4000, "stream": 3000, "stream_exact": 300, "evaluate": 600, "plan": 2000}[c["kind"]]
    c["bs"] = _log(rng, 20 if c["kind"] in ("score", "embed") else 100, min(most, room // 4))
    c["budget"] = _log(rng, 100, max(200, min(10000, (c["n_src"] + c["n_dst"]) // 4)))
    c["strategy"] = rng.choice(["MRD", "LRU", "2Q"])
    if c["kind"] != "plan":
        c["layers"] = 2 if c["kind"] == "stream_exact" else rng.choice([1, 2, 2, 2])
    if c["kind"] not in ("score", "embed"):
        batches = {"stream": 50, "stream_exact": 30, "evaluate": 20, "plan": 200}[c["kind"]]
        c["edges"] = max(1, min(_log(rng, 2 * c["bs"], batches * c["bs"]), room - (WARM + 1) * c["bs"]))
    return c


# ---------------------------------------------------------------------------------------------- inputs
def _zipf(gen, m, s, n):
    """n ids in [0, m) with probability proportional to (id + 1)^-s."""
    # (summed on the host: a floating sum over the GPU's threads is not the same twice)
    cdf = torch.from_numpy(np.cumsum(np.arange(1, m + 1, dtype=np.float64) ** -s)).cuda()
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=gen) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=m - 1)


def _graph(case, gen):
    """A synthetic edge stream (ids, times on the host) drawn on the GPU, as orca_b200/synthetic.py draws its own."""
    E, ns, nd = case["n_edges"], case["n_src"], case["n_dst"]
    rand = lambda: torch.rand(E, dtype=torch.float64, device="cuda", generator=gen)
    src = 1 + _zipf(gen, ns, case["zipf_src"], E)
    if nd:
        dst = 1 + ns + _zipf(gen, nd, case["zipf_dst"], E)
    elif case["zipf_dst"]:
        dst = 1 + _zipf(gen, ns, case["zipf_dst"], E)
    else:
        # preferential attachment: four times out of five an endpoint of an earlier edge, else any node
        at = torch.arange(E, device="cuda")
        j, copy, second = (rand() * at).long(), rand() < 0.8, rand() < 0.5
        copy[0] = False
        val = torch.where(copy & ~second, src[j], 1 + (rand() * ns).long())
        ptr = torch.where(copy & second, j, torch.full_like(j, -1))
        while bool((ptr >= 0).any()):
            at = ptr.clamp(min=0)
            ready = ptr[at] < 0
            val = torch.where((ptr >= 0) & ready, val[at], val)
            ptr = torch.where((ptr >= 0) & ~ready, ptr[at], torch.full_like(ptr, -1))
        dst = val
    if not nd:
        dst = torch.where(dst == src, src % ns + 1, dst)     # no self loops
    if case["times"] == "uniform":
        ts = torch.sort(rand() * case["span"])[0]
    else:
        gap = -torch.log1p(-rand())
        if case["times"] == "bursty":
            gap *= torch.where(torch.arange(E, device="cuda") // 10000 % 2 == 0, 0.1, 1.9)
        # (summed in whole ticks, so that the sum is the same every time)
        ts = torch.cumsum((gap * 2 ** 20).long(), 0).double() * (case["span"] / E / 2 ** 20)
    seen = torch.unique(dst)
    neg = seen[(rand() * len(seen)).long()]
    return types.SimpleNamespace(n_nodes=ns + nd + 1, src=src.cpu().numpy(), dst=dst.cpu().numpy(),
                                 neg=neg.cpu().numpy(), ts=ts.cpu().numpy(), eidx=np.arange(1, E + 1))


def _part(g, lo, hi):
    return types.SimpleNamespace(sources=g.src[lo:hi], destinations=g.dst[lo:hi], timestamps=g.ts[lo:hi],
                                 edge_idxs=g.eidx[lo:hi], n_interactions=hi - lo, negatives=g.neg[lo:hi])


def _model(case, g, nf, args, gen):
    tgn = TGN(neighbor_finder=nf, node_features=None, edge_features=np.zeros((1, D), np.float32), device="cuda",
              n_layers=case["layers"], n_heads=2, dropout=0.1, use_memory=True, node_dimension=D, time_dimension=D,
              memory_dimension=D, embedding_module_type="graph_attention", message_function="identity",
              aggregator_type="last", memory_updater_type="gru", n_neighbors=case["k"], args=args)
    normal = lambda n: torch.randn(n, D, device="cuda", generator=gen)
    # the edge features are drawn where they are used (row 0 belongs to the padding edge)
    tgn.edge_raw_features = normal(case["n_edges"] + 1)
    tgn.edge_raw_features[0] = 0
    sd = {k: torch.from_numpy(v) for k, v in params.random_state_dict(case["layers"], seed=case["seed"]).items()}
    sd["embedding_module.time_encoder.w.weight"] = sd["time_encoder.w.weight"]
    sd["embedding_module.time_encoder.w.bias"] = sd["time_encoder.w.bias"]
    tgn.load_state_dict(sd)
    tgn.eval()
    # tables as a long run leaves them: every node has a memory, a last update before the stretch and, with two
    # layers, a historical embedding
    tgn.memory.memory.copy_(normal(g.n_nodes) * 0.4)
    tgn.memory.last_update.copy_(torch.rand(g.n_nodes, device="cuda", generator=gen) * float(g.ts[len(g.ts) // 2]))
    if case["layers"] == 2:
        tgn.embedding_module.histories[0].emb.copy_(normal(g.n_nodes))
    return tgn


def prepare(case, seed):
    case = dict(case, seed=seed % (1 << 31))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    g = _graph(case, gen)
    s = types.SimpleNamespace(kind=case["kind"], case=case, g=g)
    if case["kind"] == "adjacency":
        s.data = _part(g, 0, case["n_edges"])
        return s
    s.nf = get_neighbor_finder(_part(g, 0, case["n_edges"]), max_node_idx=g.n_nodes - 1)
    if case["kind"] == "neighbors":
        at = torch.randint(0, case["n_edges"], (case["queries"],), device="cuda", generator=gen).cpu().numpy()
        s.nodes, s.times = np.where(at % 2 == 0, g.src[at], g.dst[at]), g.ts[at]
        return s
    bs = case["bs"]
    n = case.get("edges", bs)
    s.args = argparse.Namespace(bs=bs, n_degree=case["k"], budget=case["budget"], reuse=True, gradient=False,
                                n_nodes=g.n_nodes, n_edges=case["n_edges"] + 1)
    lo = case["n_edges"] // 2
    if case["kind"] == "plan":
        s.data = _part(g, lo, lo + n)
        return s
    # the stretch to score is preceded by the batches that the model has scored when it gets there
    plan = get_cache_plan(s.args, _part(g, lo, lo + WARM * bs + n), s.nf, g.n_nodes, case["strategy"], seed=case["seed"])
    s.tgn = _model(case, g, s.nf, s.args, gen)
    before = _part(g, lo, lo + WARM * bs)
    s.data, s.plan = _part(g, lo + WARM * bs, lo + WARM * bs + n), plan[WARM:]
    s.reuse = case["kind"] != "stream_exact"
    s.tgn.eval_epoch(before.sources, before.destinations, before.negatives, before.timestamps, before.edge_idxs,
                     case["k"], bs, plan[:WARM], reuse=s.reuse)
    if case["kind"] == "evaluate":
        s.sampler = RandEdgeSampler(g.src, g.dst, seed=case["seed"])
    return s


# ---------------------------------------------------------------------------------------------- one pass
def _with_state(tgn, out):
    """What a pass returns and what it changes: the scores, the node memory and the historical embeddings."""
    m = tgn.memory
    out.update(memory=m.memory, last_update=m.last_update, messages=m.messages, message_times=m.timestamps)
    if tgn.n_layers == 2:
        out.update(history=tgn.embedding_module.histories[0].emb, cached=tgn.embedding_module.histories[0].cache_flag_dev)
    return out


def run(state):
    c, kind = state.case, state.kind
    if kind == "adjacency":
        nf = get_neighbor_finder(state.data, max_node_idx=state.g.n_nodes - 1)
        return {"indptr": nf.indptr, "neighbors": nf.adj_nbr, "edges": nf.adj_eid, "times": nf.adj_ts}
    if kind == "neighbors":
        return state.nf.get_temporal_neighbor(state.nodes, state.times, c["k"])
    if kind == "plan":
        plan = get_cache_plan(state.args, state.data, state.nf, state.g.n_nodes, c["strategy"], seed=c["seed"])
        # one array per batch, at most the budget's entries each: put into one of a size that the case gives
        nodes, n = np.zeros(len(plan) * c["budget"], dtype=np.int64), sum(len(p) for p in plan)
        np.concatenate(plan, out=nodes[:n])
        return {"sizes": np.array([len(p) for p in plan]), "nodes": nodes}
    d, tgn = state.data, state.tgn
    if kind == "score":
        pos, neg = tgn.compute_edge_probabilities(d.sources, d.destinations, d.negatives, d.timestamps, d.edge_idxs,
                                                  c["k"], True, False, state.plan[0])
        return _with_state(tgn, {"pos": pos, "neg": neg})
    if kind == "embed":
        src, dst, neg = tgn.compute_temporal_embeddings(d.sources, d.destinations, d.negatives, d.timestamps,
                                                        d.edge_idxs, c["k"], True, False, state.plan[0])
        return _with_state(tgn, {"src": src, "dst": dst, "neg": neg})
    if kind == "evaluate":
        ap, auc, acc = eval_edge_prediction(tgn, state.sampler, d, c["k"], c["bs"], cache_plan=state.plan)
        return _with_state(tgn, {"ap": float(ap), "auc": float(auc), "acc": float(acc)})
    pos, neg = tgn.eval_epoch(d.sources, d.destinations, d.negatives, d.timestamps, d.edge_idxs, c["k"], c["bs"],
                              state.plan, reuse=state.reuse)
    return _with_state(tgn, {"pos": pos, "neg": neg})


# ---------------------------------------------------------------------------------------------- what it takes
def _distinct(m, s, n):
    """Expected number of distinct ids among n draws of a Zipf(s) law over m ids (s = 0: uniform)."""
    p = np.arange(1, m + 1, dtype=np.float64) ** -s
    p /= p.sum()
    return float(-np.expm1(n * np.log1p(-np.minimum(p, 1 - 1e-12))).sum())


def work(case):
    kind, E, n_nodes = case["kind"], case["n_edges"], case["n_src"] + case["n_dst"] + 1
    if kind == "adjacency":       # (source, destination, edge id, time) of every edge in, two CSR entries out
        return {"bytes": E * 32 + 2 * E * 16 + 8 * (n_nodes + 1), "flops": 0}
    k = case["k"]
    if kind == "neighbors":       # a node and a time in, k entries (id, edge, time) read, k entries written
        q = case["queries"]
        return {"bytes": q * 12 + q * k * 16 + q * k * 12, "flops": 0}
    bs = case["bs"]
    n = case.get("edges", bs)
    nb = n / bs
    if kind == "plan":            # the endpoints and their neighbours in, the plan out
        return {"bytes": 2 * n * 12 + 2 * n * k * 16 + nb * min(case["budget"], n_nodes) * 8, "flops": 0}
    # distinct nodes of a batch: their k neighbour and edge rows are read once, their memory once; the edge rows
    # serve both layers, the neighbours' rows are the memory in layer 1 and the history in layer 2
    n_src, n_dst = case["n_src"], case["n_dst"] or case["n_src"]
    pos = _distinct(n_src, case["zipf_src"], bs) + _distinct(n_dst, case["zipf_dst"], bs)
    nodes = pos + _distinct(n_dst, 0.0, bs)
    layers = case["layers"]
    rows = nodes * k * (1 + layers) + nodes
    if kind == "stream_exact":
        rows = nodes * k * 2 + nodes * k * k
    rows += pos * (4 + 4 + 1 + 1)            # messages written and read again, memory rows written
    if layers == 2:
        rows += nodes                        # history rows written
    if kind == "embed":
        rows += 3 * bs
    per_row = 2 * D * 2 * 3 * D + 2 * 2 * 2 * k * 3 * D + 2 * (7 * D) * D + 2 * D * D   # query, attention, output
    q_rows = 3 * bs * layers if kind != "stream_exact" else 3 * bs * (2 + k)
    flops = q_rows * per_row + 2 * pos * 5 * D * 3 * D + 2 * bs * 2 * (2 * D * D + D)
    return {"bytes": nb * (rows * ROW + bs * 24), "flops": nb * flops}


def tolerance(case):
    if case["kind"] in ("adjacency", "neighbors", "plan"):
        return "exact"
    # The projections take their operands as two bf16 parts (about 16 bits) and add in 32 bits; against all-fp32
    # products this leaves up to 1e-5 of the results' norm, over both layers and the memory handed from batch to batch.
    if case["kind"] == "evaluate":
        return {"rel": 1e-3, "max": 4e-3}     # (metrics of ranks: the ranks of close scores may swap)
    return {"rel": 5e-5, "max": 1e-3}
