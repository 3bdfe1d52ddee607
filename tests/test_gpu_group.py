"""Groups of batches (TGN.eval_epoch on one GPU) against one call per batch: the same bits in the scores and in every
state table, for each recursion, for batch sizes from one edge to more than a tile, for streams that end inside a
group, at a group's last batch and with a short batch, and for a second epoch on the same buffers."""
import numpy as np
import pytest
import torch

from helpers import graph
from orca_b200 import synthetic

pytestmark = pytest.mark.gpu


def _plan(g, bs, k, budget, strategy, E):
    import argparse
    import types
    from orca_b200.cache import get_cache_plan
    from orca_b200.neighbor_finder import get_neighbor_finder
    nf = get_neighbor_finder(g)
    data = types.SimpleNamespace(sources=g.sources[:E], destinations=g.destinations[:E], timestamps=g.timestamps[:E])
    return get_cache_plan(argparse.Namespace(bs=bs, n_degree=k, budget=budget), data, nf, g.n_nodes, strategy)


# (graph, batch size, k, edges, recursion, layers)
CASES = [("t_nb2", 37, 10, 5011, "budget", 2),       # 136 batches: five groups, the last batch short
         ("t_bip2", 64, 5, 64 * 64, "budget", 2),    # two full groups
         ("t_2q", 1, 10, 70, "budget", 2),           # one edge a batch
         ("t_lru", 300, 20, 5999, "budget", 2),      # k above 16; more rows than a tile of either kernel
         ("t_nb2", 1500, 3, 5000, "budget", 2),      # three batches and a bit
         ("t_nb2", 50, 10, 2030, "all", 2),          # unlimited reuse
         ("t_nb2", 50, 10, 2030, "none", 2),         # no reuse: a layer-1 row per sampled neighbour
         ("t_lru", 33, 20, 700, "none", 2),
         ("c1", 129, 10, 6000, "budget", 1),
         ("c1", 600, 10, 20000, "budget", 2),        # groups whose last updates leave the memory chain
         ("c1", 512, 10, 16400, "budget", 2)]        # a group without, then one with


@pytest.mark.parametrize("name,bs,k,E,recursion,layers", CASES)
def test_group_equals_batches(name, bs, k, E, recursion, layers):
    import dataclasses
    from test_gpu_model import make_model
    g = graph(name)
    budget = 0 if recursion == "all" else g.spec.budget
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, bs=bs, n_degree=k, n_layers=layers, budget=budget))
    neg = synthetic.negative_destinations(g, seed=1)
    plan = _plan(g, bs, k, g.spec.budget, g.spec.strategy, E) if recursion == "budget" else None
    a, b = make_model(g), make_model(g)
    reuse = recursion != "none"
    nb = -(-E // bs)
    for epoch in range(2):
        pos, ngs = [], []
        for i in range(nb):
            sl = slice(i * bs, min(E, (i + 1) * bs))
            p, q = a.compute_edge_probabilities(g.sources[sl], g.destinations[sl], neg[sl], g.timestamps[sl],
                                                g.edge_idxs[sl], k, reuse, False, plan[i] if plan else None)
            pos.append(p.cpu().numpy().ravel()), ngs.append(q.cpu().numpy().ravel())
        ca = a.check_status()
        p2, q2 = b.eval_epoch(g.sources[:E], g.destinations[:E], neg[:E], g.timestamps[:E], g.edge_idxs[:E], k, bs, plan,
                              reuse=reuse)
        cb = b.check_status()
        assert np.array_equal(np.concatenate(pos), p2) and np.array_equal(np.concatenate(ngs), q2), epoch
        if recursion == "budget" and layers == 2:
            assert ca[:2] == cb[:2]
        for t in ("memory", "last_update", "messages", "timestamps", "nodes_dev"):
            assert torch.equal(getattr(a.memory, t), getattr(b.memory, t)), (epoch, t)
        if layers == 2:
            ha, hb = a.embedding_module.histories[0], b.embedding_module.histories[0]
            assert torch.equal(ha.emb, hb.emb) and torch.equal(ha.cache_flag_dev, hb.cache_flag_dev)


@pytest.mark.parametrize("budget,chunks", [(1, "several"), (1500, "one")])
def test_rows_that_share_features_equal_batches(budget, chunks):
    """Layer 1 of a group computes what depends on a row's own features once per distinct memory row if the group's rows fit
    one chunk, and per row otherwise (next to nothing is cached: the recomputed rows outnumber the batches' own).  Either
    way the scores and tables are those of the single batches, whose rows share nothing."""
    import argparse
    import dataclasses
    import types
    from orca_b200.cache import get_cache_plan
    from test_gpu_model import make_model
    g = graph("c1")
    bs, k, E = 100, 20, 3000
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, bs=bs, n_degree=k, n_layers=2, budget=budget))
    neg = synthetic.negative_destinations(g, seed=1)
    lo = len(g.sources) - E
    part = lambda x, a, b: x[lo + a:lo + b]
    data = types.SimpleNamespace(sources=part(g.sources, 0, E), destinations=part(g.destinations, 0, E),
                                 timestamps=part(g.timestamps, 0, E))
    m = make_model(g)
    nf = m.embedding_module.neighbor_finder
    plan = get_cache_plan(argparse.Namespace(bs=bs, n_degree=k, budget=budget), data, nf, g.n_nodes, "MRD")
    one, rows = [], 0
    for i in range(E // bs):
        a = [part(x, i * bs, (i + 1) * bs) for x in (g.sources, g.destinations, neg, g.timestamps, g.edge_idxs)]
        one.append(torch.cat(m.compute_edge_probabilities(*a, k, True, False, plan[i])).cpu().numpy().ravel())
        rows += m.check_status()[0]
    assert (rows > 3 * E + 3 * E // 4) == (chunks == "several")
    b = make_model(g)
    p, q = b.eval_epoch(*[part(x, 0, E) for x in (g.sources, g.destinations, neg, g.timestamps, g.edge_idxs)], k, bs, plan)
    one = np.stack(one).reshape(-1, 2, bs)
    assert np.array_equal(one[:, 0].ravel(), p) and np.array_equal(one[:, 1].ravel(), q)
    for t in ("memory", "last_update", "messages"):
        assert torch.equal(getattr(m.memory, t), getattr(b.memory, t)), t
    assert torch.equal(m.embedding_module.histories[0].emb, b.embedding_module.histories[0].emb)


def test_groups_of_one_large_batch_equal_batches():
    """A batch that fills a group alone, with enough updates that the last of every node leave the memory chain."""
    test_group_equals_batches("c1", 9000, 10, 18500, "budget", 2)


def test_a_stream_that_fails_leaves_a_model_that_works(monkeypatch):
    """A stream can fail in the middle -- here an id that cannot be packed, in the third group, and a workspace that
    cannot be allocated.  What was enqueued has finished when the error is raised, and the next stream runs as on a
    fresh model."""
    from test_gpu_model import make_model
    g = graph("t_nb2")
    bs, k, E = 20, 10, 2000
    neg = synthetic.negative_destinations(g, seed=1)
    plan = _plan(g, bs, k, g.spec.budget, g.spec.strategy, E)
    m, fresh = make_model(g), make_model(g)
    run = lambda model, plan, n, k=k: model.eval_epoch(g.sources[:n], g.destinations[:n], neg[:n], g.timestamps[:n],
                                                       g.edge_idxs[:n], k, bs, plan)
    state = [t.clone() for t in m.memory.backup_memory()]
    waits = []
    synchronize = torch.cuda.synchronize
    monkeypatch.setattr(torch.cuda, "synchronize", lambda *a: (waits.append(a), synchronize(*a))[1])
    bad = list(plan)
    bad[70] = ["not an id"] * len(plan[70])
    with pytest.raises(ValueError):
        run(m, bad, E)
    assert waits
    del waits[:]
    with pytest.raises(Exception):
        run(m, plan, E, k=33)              # (no workspace for more than 32 neighbours)
    assert waits
    m.memory.restore_memory(state)
    m.embedding_module.reset_history()
    m.embedding_module.histories[0].cache_flag = np.zeros(g.n_nodes)
    for a, b in zip(run(m, plan, E), run(fresh, plan, E)):
        assert np.array_equal(a, b)
    assert torch.equal(m.memory.memory, fresh.memory.memory)


@pytest.mark.parametrize("bs,E", [(1, 40), (255, 700), (256, 1024), (257, 1000), (4096, 9000), (5000, 9000)])
def test_metrics_on_the_device_equal_the_hosts(bs, E):
    """eval_epoch_metrics against orca_link_metrics over the scores of the same stream, on both sides of a part's 256
    edges and of the largest batch that is evaluated on the device; with scores that are equal (nodes that a fresh model
    knows nothing of)."""
    import dataclasses
    from orca_b200 import _lib
    from test_gpu_model import make_model
    g = graph("c1")
    k = g.spec.n_degree
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, bs=bs))
    neg = synthetic.negative_destinations(g, seed=1)
    args = (g.sources[:E], g.destinations[:E], neg[:E], g.timestamps[:E], g.edge_idxs[:E], k, bs)
    pos, ngs = make_model(g).eval_epoch(*args)
    assert len(np.unique(pos)) < E or bs == 1
    want = np.empty((-(-E // bs), 3))
    assert _lib.lib().orca_link_metrics(pos.ctypes.data, ngs.ctypes.data, E, bs, want.ctypes.data) == 0
    # (sums of at most bs doubles of one sign in another order: bs * 2^-53)
    np.testing.assert_allclose(make_model(g).eval_epoch_metrics(*args), want, rtol=1e-12)


@pytest.mark.parametrize("bs", [256, 300, 4096, 4200])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_metrics_of_scores_that_are_not_finite_are_refused(bs, bad):
    """A memory row that is not finite makes the scores of its node's edges NaN.  The metrics are refused with the batch's
    number, as the host's are, whether they are made on the device (up to 4096 edges a batch) or not."""
    import dataclasses
    from orca_b200 import _lib
    from test_gpu_model import make_model
    g = graph("c1")
    E = 2 * bs
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, bs=bs))
    args = (g.sources[:E], g.destinations[:E], synthetic.negative_destinations(g, seed=1)[:E], g.timestamps[:E],
            g.edge_idxs[:E], g.spec.n_degree, bs)
    node = int(np.setdiff1d(g.sources[bs:E], np.r_[g.sources[:bs], g.destinations[:bs], args[2][:bs]])[0])
    said = []
    for metrics in (False, True):
        m = make_model(g)
        m.memory.memory[node] = bad
        if metrics:
            with pytest.raises(ValueError) as e:
                m.eval_epoch_metrics(*args)
            said.append(str(e.value))
        else:
            pos, neg = m.eval_epoch(*args)
            assert np.isnan(pos).any() and np.isfinite(pos).any()
            assert _lib.lib().orca_link_metrics(pos.ctypes.data, neg.ctypes.data, E, bs, np.empty((2, 3)).ctypes.data) == 1
            said.append(_lib.lib().orca_last_error().decode())
    assert said[0] == said[1]


@pytest.mark.parametrize("bs,k", [(2730, 32), (2731, 32), (2731, 1), (5462, 17)])
def test_calls_that_order_more_rows_than_are_kept(bs, k):
    """A call's rows are handed out in the order of their valid slots, which is kept for 8192 rows and counted again beyond."""
    test_group_equals_batches("c1", bs, k, 2 * bs + 100, "budget", 2)
