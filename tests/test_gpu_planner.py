"""The device planners (orca_plan_device: MRD, LRU, 2Q) against the reference's plans (golden fixtures) and
against the oracle's planner on inputs that put many equal keys at the budget line, where the order numba's
argsort leaves among equal keys -- and, for LRU and 2Q, the stream of its Mersenne Twister -- decide which
nodes stay cached.  Plans are compared entry by entry, in order; the statistics are compared as integers."""
import dataclasses

import numpy as np
import pytest
import torch

from helpers import golden, graph, unpack

pytestmark = pytest.mark.gpu


def _device_plan(g, bs, k, budget, tables_from_oracle=True, strategy="MRD", seed=0):
    """Plan of the device planner; the neighbour table comes from the oracle's sampler (so that the test
    isolates the planner) or from the product sampler."""
    from oracle import tgn_oracle
    from orca_b200 import cache
    nodes, ts = cache.batch_query_order(g.sources, g.destinations, g.timestamps, bs)
    adj = tgn_oracle.Adjacency(g.sources, g.destinations, g.edge_idxs, g.timestamps, g.n_nodes)
    if tables_from_oracle:
        nbr = torch.as_tensor(tgn_oracle.sample_neighbors(adj, nodes, ts, k)[0].astype(np.int32)).cuda()
    else:
        from orca_b200.neighbor_finder import get_neighbor_finder
        nbr = get_neighbor_finder(g, g.n_nodes - 1, device="cuda").sample_device(nodes, ts, k)[0]
    plan, stats = cache.plan_device(strategy, torch.as_tensor(nodes).cuda(), nbr, g.n_edges, bs, k, g.n_nodes, budget,
                                    seed)
    return adj, plan, stats


@pytest.mark.parametrize("case", ["c1", "t_bip2", "t_nb2", "t_lru", "t_2q"])
@pytest.mark.parametrize("strategy", ["MRD", "LRU", "2Q"])
def test_plans_match_reference(case, strategy):
    gold = golden(case)
    g = graph(str(gold["spec"]))
    _, got, _ = _device_plan(g, g.spec.bs, g.spec.n_degree, g.spec.budget, tables_from_oracle=False,
                             strategy=strategy)
    want = unpack(gold[f"plan_{strategy}_flat"], gold[f"plan_{strategy}_off"])
    assert len(got) == len(want)
    for b, (a, w) in enumerate(zip(got, want)):
        assert a.dtype == np.int64 and np.array_equal(a, w), f"batch {b}"


@pytest.mark.parametrize("budget,bs,seed", [(7, 50, 1), (40, 120, 2), (300, 200, 3), (2, 64, 4), (1000, 400, 5),
                                            (100000, 200, 6), (200000, 200, 7)])
@pytest.mark.parametrize("strategy", ["MRD", "LRU", "2Q"])
def test_plans_match_oracle_on_tight_budgets(strategy, budget, bs, seed):
    """Budgets from far below to far above the number of candidates; statistics included.  (The last budget
    makes the candidate capacity larger than a thread-block cluster takes, so the one-CTA kernels run.)"""
    from oracle import planner
    from orca_b200 import synthetic
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], n_src=400, n_edges=3000, bs=bs, budget=budget)
    g = synthetic.make_graph(spec, seed=seed)
    adj, got, stats = _device_plan(g, bs, 10, budget, strategy=strategy, seed=seed)
    rb = planner.read_batches(g.sources, g.destinations, g.timestamps, bs, 10, adj, g.n_nodes)
    want, wstats = planner.solve(strategy, rb, g.n_nodes, budget, seed=seed)
    assert len(got) == len(want)
    for b, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w), f"batch {b}"
    assert (int(stats[0]), int(stats[1])) == wstats[:2]
    if wstats[0]:
        assert stats[2] / stats[0] == wstats[2]


def test_mrd_long_ranges_of_equal_keys():
    """A wide graph with large batches: tens of thousands of candidates per batch, nearly all with the key
    of "not needed again as a neighbour", cut by a budget in the middle of them -- every level of the
    partition emulation is exercised, over many ranges at once."""
    from oracle import planner
    from orca_b200 import synthetic
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], n_src=60000, n_edges=60000, bs=2000,
                               budget=9000)
    g = synthetic.make_graph(spec, seed=11)
    adj, got, stats = _device_plan(g, spec.bs, 10, spec.budget)
    rb = planner.read_batches(g.sources, g.destinations, g.timestamps, spec.bs, 10, adj, g.n_nodes)
    want, wstats = planner.solve("MRD", rb, g.n_nodes, spec.budget)
    assert max(len(w) for w in want) == spec.budget
    for b, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w), f"batch {b}"
    assert (int(stats[0]), int(stats[1])) == wstats[:2]


@pytest.mark.parametrize("strategy", ["MRD", "LRU", "2Q"])
@pytest.mark.parametrize("n_src,n_edges,bs,budget", [(3000, 30000, 600, 1200),     # lists of one entry a thread
                                                     (60000, 60000, 2000, 24000),  # MRD: some fit shared memory
                                                     (60000, 40000, 2000, 9000),   # of up to twenty
                                                     (60000, 60000, 4000, 44000),  # longer than shared memory takes
                                                     (400000, 20000, 1000, 2000)])  # bitmaps in global memory
def test_plans_at_the_limits_of_shared_memory(strategy, n_src, n_edges, bs, budget):
    from oracle import planner
    from orca_b200 import synthetic
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], n_src=n_src, n_edges=n_edges, bs=bs, budget=budget)
    g = synthetic.make_graph(spec, seed=12)
    adj, got, stats = _device_plan(g, bs, 20, budget, strategy=strategy, seed=9)
    rb = planner.read_batches(g.sources, g.destinations, g.timestamps, bs, 20, adj, g.n_nodes)
    want, wstats = planner.solve(strategy, rb, g.n_nodes, budget, seed=9)
    for b, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w), f"batch {b}"
    assert (int(stats[0]), int(stats[1])) == wstats[:2]


@pytest.mark.parametrize("strategy", ["LRU", "2Q"])
@pytest.mark.parametrize("n_nodes", [65536, 65537])
@pytest.mark.parametrize("budget", [900, 30000])
def test_plans_where_the_listing_of_sets_changes(strategy, n_nodes, budget):
    """Sets of up to 65,536 nodes are listed by half words, larger ones by words; with the larger budget nothing is evicted."""
    from oracle import planner
    from orca_b200 import synthetic
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], n_src=n_nodes - 1, n_edges=12000, bs=600, budget=budget)
    g = synthetic.make_graph(spec, seed=13)
    assert g.n_nodes == n_nodes
    adj, got, stats = _device_plan(g, 600, 10, budget, strategy=strategy, seed=9)
    rb = planner.read_batches(g.sources, g.destinations, g.timestamps, 600, 10, adj, g.n_nodes)
    want, wstats = planner.solve(strategy, rb, g.n_nodes, budget, seed=9)
    assert len(got) == len(want)
    for b, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w), f"batch {b}"
    assert (int(stats[0]), int(stats[1])) == wstats[:2]


def test_plan_buffer_too_small_is_reported():
    from orca_b200 import _lib, cache
    g = graph("t_nb2")
    bs, k, budget = g.spec.bs, g.spec.n_degree, 50
    nodes, ts = cache.batch_query_order(g.sources, g.destinations, g.timestamps, bs)
    from orca_b200.neighbor_finder import get_neighbor_finder
    nbr = get_neighbor_finder(g, g.n_nodes - 1, device="cuda").sample_device(nodes, ts, k)[0]
    L = _lib.lib()
    ws_bytes = L.orca_plan_mrd_workspace_bytes(g.n_edges, bs, k, g.n_nodes, budget)
    ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
    nd = torch.as_tensor(nodes).cuda()
    flat = torch.empty(60, dtype=torch.int32, device="cuda")
    off = torch.zeros(g.n_batches + 1, dtype=torch.int64, device="cuda")
    stats = torch.zeros(3, dtype=torch.int64, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    _lib.check(L.orca_plan_mrd(nd.data_ptr(), g.n_edges, bs, k, nbr.data_ptr(), g.n_nodes, budget, flat.data_ptr(), 60,
                               off.data_ptr(), stats.data_ptr(), status.data_ptr(), ws.data_ptr(), ws_bytes,
                               _lib.stream_ptr(torch.device("cuda"))))
    torch.cuda.synchronize()
    assert int(status[0]) == 4        # ORCA_E_CAPACITY
    with pytest.raises(_lib.OrcaError):
        # the same call with too small a workspace is refused on the host
        _lib.check(L.orca_plan_mrd(nd.data_ptr(), g.n_edges, bs, k, nbr.data_ptr(), g.n_nodes, budget,
                                   flat.data_ptr(), 60, off.data_ptr(), stats.data_ptr(), status.data_ptr(),
                                   ws.data_ptr(), ws_bytes - 1, _lib.stream_ptr(torch.device("cuda"))))


@pytest.mark.parametrize("E,bs", [(1, 1), (7, 7), (1000, 300), (101, 100), (250001, 2000), (3, 10)])
def test_queries_on_the_device_are_in_batch_order(E, bs):
    from orca_b200 import cache
    rs = np.random.RandomState(E)
    src, dst, ts = rs.randint(1, 1 << 30, E), rs.randint(1, 1 << 30, E), rs.rand(E)
    want = cache.batch_query_order(src, dst, ts, bs)
    got = cache._queries_device(src, dst, ts, bs, torch.device("cuda"))
    assert all(np.array_equal(g.cpu().numpy(), w) for g, w in zip(got, want))


@pytest.mark.parametrize("on_host", [False, True])
def test_columns_of_a_plan_may_be_longer_than_the_sources_but_not_shorter(on_host, monkeypatch):
    """`sources` says how many edges there are, whichever way the queries take to the device."""
    import argparse
    import types
    from orca_b200 import cache
    from orca_b200.neighbor_finder import NeighborFinder, get_neighbor_finder
    g = graph("t_nb2")
    if on_host:
        monkeypatch.setattr(NeighborFinder, "PINNED_TABLE", 16)
    nf, args = get_neighbor_finder(g), argparse.Namespace(bs=100, n_degree=10, budget=50)
    plan = lambda n, m, t: cache.get_cache_plan(args, types.SimpleNamespace(
        sources=g.sources[:n], destinations=g.destinations[:m], timestamps=g.timestamps[:t]), nf, g.n_nodes, "LRU")
    want = plan(950, 950, 950)
    for more in ((950, 1000, 950), (950, 950, 951), (950, 1200, 1000)):
        got = plan(*more)
        assert len(got) == len(want) and all(np.array_equal(a, w) for a, w in zip(got, want)), more
    for fewer in ((950, 940, 950), (950, 950, 300)):
        with pytest.raises(ValueError):
            plan(*fewer)
    as_lists = cache._queries_device(list(g.sources[:950]), g.destinations[:950].astype(np.int32),
                                     g.timestamps[:950].astype(np.float32), 100, torch.device("cuda"))
    host = cache.batch_query_order(g.sources[:950], g.destinations[:950], g.timestamps[:950].astype(np.float32), 100)
    assert all(np.array_equal(a.cpu().numpy(), w) for a, w in zip(as_lists, host))


@pytest.mark.parametrize("strategy", ["MRD", "LRU", "2Q"])
def test_a_plan_covers_the_nodes_of_its_graph_whatever_number_is_given(strategy):
    """A number of nodes below the graph's (one short, as without the padding node, or far off) must not make the planners
    reach outside their tables."""
    import argparse
    from orca_b200 import cache
    from orca_b200.neighbor_finder import get_neighbor_finder
    g = graph("t_nb2")
    nf, args = get_neighbor_finder(g), argparse.Namespace(bs=100, n_degree=10, budget=50)
    seen = []
    plan_device = cache.plan_device
    cache_plan = lambda n: cache.get_cache_plan(args, g, nf, n, strategy)
    try:
        cache.plan_device = lambda *a: (seen.append(a[6]), plan_device(*a))[1]
        want = cache_plan(g.n_nodes)
        for n in (g.n_nodes - 1, 10, g.n_nodes + 70000):
            got = cache_plan(n)
            assert len(got) == len(want) and all(np.array_equal(a, w) for a, w in zip(got, want)), n
    finally:
        cache.plan_device = plan_device
    assert seen == [g.n_nodes] * 3 + [g.n_nodes + 70000]


@pytest.mark.parametrize("strategy", ["MRD", "LRU", "2Q"])
@pytest.mark.parametrize("n_src", [130000, 700000])      # sets in shared memory and in global memory
def test_plans_of_several_launches(n_src, strategy):
    """The lists of 135 batches of 2000 edges with 30 neighbours lie in memory at a time (LRU, 2Q): two full launches and one
    of a short batch.  Against the host's policies over the same tables."""
    from orca_b200 import cache, synthetic
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], n_src=n_src, n_edges=541001, bs=2000, budget=3000)
    g = synthetic.make_graph(spec, seed=13)
    nodes, ts = cache.batch_query_order(g.sources, g.destinations, g.timestamps, 2000)
    from orca_b200.neighbor_finder import get_neighbor_finder
    nbr = get_neighbor_finder(g, g.n_nodes - 1).sample_device(nodes, ts, 30)[0]
    got, stats = cache.plan_device(strategy, torch.as_tensor(nodes).cuda(), nbr, g.n_edges, 2000, 30, g.n_nodes, 3000, seed=4)
    want, wstats = cache.plan_from_tables(strategy, g.sources, g.destinations, 2000, 30, nbr.cpu().numpy(), g.n_nodes, 3000,
                                          seed=4)
    assert len(got) == len(want) == 271 and max(map(len, want)) > 2000
    for b, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w), f"batch {b}"
    assert np.array_equal(stats, wstats)


def test_mrd_plan_with_more_lists_than_there_is_room_for():
    """15,000 nodes met evenly: nearly every entry of a batch's table is another node, 17 M and more in all.  The kernels that
    need no lists make the plan."""
    from orca_b200 import cache
    from orca_b200.neighbor_finder import NeighborFinder
    rs = np.random.RandomState(3)
    E, n, bs, k, budget = 500000, 15000, 50, 32, 400
    src, dst, ts = rs.randint(1, n, E), rs.randint(1, n, E), np.arange(E, dtype=np.float64)
    nf = NeighborFinder.build_on_device(src, dst, np.arange(1, E + 1), ts, n)
    nodes, t = cache.batch_query_order(src, dst, ts, bs)
    nbr = nf.sample_device(nodes, t, k)[0]
    table = nbr.cpu().numpy().reshape(E // bs, -1)
    assert sum(len(np.unique(r)) for r in table) > 16 << 20
    got, stats = cache.plan_device("MRD", torch.as_tensor(nodes).cuda(), nbr, E, bs, k, n, budget)
    want, wstats = cache.plan_from_tables("MRD", src, dst, bs, k, nbr.cpu().numpy(), n, budget)
    assert len(got) == len(want)
    for b, (a, w) in enumerate(zip(got, want)):
        assert np.array_equal(a, w), f"batch {b}"
    assert np.array_equal(stats, wstats)


def test_plans_that_callers_keep_hold_a_bounded_amount_of_page_locked_memory(monkeypatch):
    """A plan of 2 MB or more stays in the page-locked memory that it was copied to, for as long as one of its batches is
    held; beyond the limit on what callers hold, and below 2 MB, plans are ordinary arrays with the same contents."""
    import gc
    from orca_b200 import cache
    from orca_b200.neighbor_finder import NeighborFinder, _Lent
    monkeypatch.setattr(NeighborFinder, "LENT", _Lent(16 << 20))
    rs = np.random.RandomState(2)
    locked = lambda a: torch.from_numpy(a).is_pinned()
    for n, share in (((2 << 20) // 8 - 1, 0), ((2 << 20) // 8, 2 << 20), (400000, 4 << 20), (3 << 20, None)):
        ids = rs.randint(0, 1 << 31, n).astype(np.int32)
        d_ids = torch.from_numpy(ids).cuda()
        held = [cache._ids_to_host(d_ids)[n // 2:] for _ in range(10)]      # (a batch of each keeps all of it)
        gc.collect()
        want = 0 if not share else min(10, (16 << 20) // share)
        assert [locked(a) for a in held] == [True] * want + [False] * (10 - want), n
        for a in held:
            assert a.dtype == np.int64 and np.array_equal(a, ids[n // 2:])
        del held, a
        gc.collect()
