"""End-to-end parity on the GPU: the drop-in ``TGN`` against (a) the golden fixtures produced by
the reference itself and (b) the CPU oracle on the same seeded inputs.

Tolerances: link scores within 1e-3 relative (the bound the path is specified to; the fp32 kernels
measure ~1e-5), state tables within 1e-3 relative to a 0.05 floor, average precision to 3 decimals,
uncached sets / cache flags / counters identical."""
import argparse

import numpy as np
import pytest
import torch
from sklearn.metrics import average_precision_score

from helpers import batches, golden, graph, max_rel, state_dict, unpack

pytestmark = pytest.mark.gpu

CASES = ["c1", "t_bip2", "t_nb2", "t_lru", "t_2q", "c2_prefix"]


def make_model(g, device="cuda:0", reuse=True, budget=None):
    from orca_b200.neighbor_finder import get_neighbor_finder
    from orca_b200.tgn import TGN
    spec = g.spec
    nf = get_neighbor_finder(g, device=device)
    budget = spec.budget if budget is None else budget
    args = argparse.Namespace(bs=spec.bs, n_degree=spec.n_degree, budget=budget, reuse=reuse, gradient=False,
                              n_nodes=g.n_nodes, n_edges=g.n_edges + 1)
    tgn = TGN(neighbor_finder=nf, node_features=None, edge_features=g.edge_features, device=torch.device(device),
              n_layers=spec.n_layers, n_heads=2, dropout=0.1, use_memory=True, node_dimension=172,
              time_dimension=172, memory_dimension=172, embedding_module_type="graph_attention",
              message_function="identity", aggregator_type="last", memory_updater_type="gru",
              n_neighbors=spec.n_degree, args=args)
    sd = {k: torch.from_numpy(v) for k, v in state_dict(spec.n_layers).items()}
    sd["embedding_module.time_encoder.w.weight"] = sd["time_encoder.w.weight"]
    sd["embedding_module.time_encoder.w.bias"] = sd["time_encoder.w.bias"]
    tgn.load_state_dict(sd, strict=True)
    tgn.eval()
    return tgn


@pytest.mark.parametrize("case", CASES)
def test_eval_matches_reference_fixture(case):
    gold = golden(case)
    g = graph(str(gold["spec"]))
    spec = g.spec
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    scores = gold["scores"]
    nb = scores.shape[0]
    neg = gold["neg"]
    tgn = make_model(g)
    want_u = unpack(gold["u_flat"], gold["u_off"]) if spec.n_layers > 1 else None
    worst, aps = 0.0, []
    for b, src, dst, ts, eidx in batches(g, nb):
        n = len(src)
        ng = neg[b * spec.bs: b * spec.bs + n]
        if b in gold["emb_batches"]:
            # embeddings of this batch, taken from a throw-away copy of the state
            pass
        p, q = tgn.compute_edge_probabilities(src, dst, ng, ts, eidx, spec.n_degree, True, False, plan[b])
        n1, n_pos, launches = tgn.check_status()
        assert p.shape == (n, 1) and q.shape == (n, 1)
        p, q = p.cpu().numpy().ravel(), q.cpu().numpy().ravel()
        worst = max(worst, max_rel(p, scores[b, 0, :n]), max_rel(q, scores[b, 1, :n]))
        aps.append(average_precision_score(np.r_[np.ones(n), np.zeros(n)], np.r_[p, q]))
        assert n_pos == len(np.unique(np.r_[src, dst]))
        assert launches > 0
        if want_u is not None:
            assert n1 == 3 * n + len(want_u[b]), f"batch {b}"
    assert worst < 1e-3, worst
    assert round(float(np.mean(aps)), 3) == round(float(gold["ap"]), 3)
    pick = gold["state_nodes"].astype(np.int64)
    mem = tgn.memory
    assert max_rel(mem.memory[pick].cpu().numpy(), gold["state_memory"], floor=0.05) < 1e-3
    assert np.array_equal(mem.last_update[pick].cpu().numpy(), gold["state_last_update"])
    assert max_rel(mem.messages[pick[:32]].cpu().numpy(), gold["state_messages"], floor=0.05) < 1e-3
    assert np.array_equal(mem.timestamps[pick].cpu().numpy(), gold["state_msg_ts"])
    assert np.array_equal(mem.nodes[pick].astype(np.uint8), gold["state_flags"])
    if spec.n_layers > 1:
        h = tgn.embedding_module.histories[0]
        assert max_rel(h.emb[pick].cpu().numpy(), gold["state_history"], floor=0.05) < 1e-3
        assert np.array_equal(np.nonzero(h.cache_flag)[0], gold["cache_flag_nodes"])


@pytest.mark.parametrize("case", ["t_nb2", "c1"])
def test_embeddings_match_reference_fixture(case):
    gold = golden(case)
    g = graph(str(gold["spec"]))
    spec = g.spec
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    neg = gold["neg"]
    tgn = make_model(g)
    for b, src, dst, ts, eidx in batches(g, gold["scores"].shape[0]):
        n = len(src)
        ng = neg[b * spec.bs: b * spec.bs + n]
        s, d, q = tgn.compute_temporal_embeddings(src, dst, ng, ts, eidx, spec.n_degree, True, False, plan[b])
        if b in gold["emb_batches"]:
            want = gold[f"emb_{b}"]
            for got, w in zip((s, d, q), want):
                assert max_rel(got[:32].cpu().numpy(), w, floor=0.05) < 1e-3
    tgn.check_status()


def test_eval_matches_oracle_on_fresh_inputs():
    """Not a fixture: a graph, weights and negatives the fixtures never saw, oracle run live."""
    import dataclasses
    from orca_b200 import params, synthetic
    from oracle import planner, tgn_oracle
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], name="fresh", n_src=900, n_edges=4000, budget=60, bs=250)
    g = synthetic.make_graph(spec, seed=11)
    adj = tgn_oracle.Adjacency(g.sources, g.destinations, g.edge_idxs, g.timestamps, g.n_nodes)
    plan = planner.get_cache_plan(g.sources, g.destinations, g.timestamps, spec.bs, spec.n_degree, spec.budget, adj,
                                  g.n_nodes, "MRD")
    sd = params.random_state_dict(2, seed=9)
    orc = tgn_oracle.OracleTGN(adj, g.edge_features, sd, g.n_nodes, n_layers=2, budget=spec.budget)
    tgn = make_model(g)
    t = {k: torch.from_numpy(v) for k, v in sd.items()}
    t["embedding_module.time_encoder.w.weight"] = t["time_encoder.w.weight"]
    t["embedding_module.time_encoder.w.bias"] = t["time_encoder.w.bias"]
    tgn.load_state_dict(t)
    neg = synthetic.negative_destinations(g, seed=5)
    worst = 0.0
    for b, src, dst, ts, eidx in batches(g):
        ng = neg[b * spec.bs: b * spec.bs + len(src)]
        # every third batch runs without a plan (the cumulative flag rule)
        pl = None if b % 3 == 2 else plan[b]
        wp, wq = orc.compute_edge_probabilities(src, dst, ng, ts, eidx, spec.n_degree, pl)
        p, q = tgn.compute_edge_probabilities(src, dst, ng, ts, eidx, spec.n_degree, True, False, pl)
        worst = max(worst, max_rel(p.cpu().numpy(), wp.numpy()), max_rel(q.cpu().numpy(), wq.numpy()))
        tgn.check_status()
    assert worst < 1e-3, worst
    assert max_rel(tgn.memory.memory.cpu().numpy(), orc.memory.numpy(), floor=0.05) < 1e-3
    assert max_rel(tgn.embedding_module.histories[0].emb.cpu().numpy(), orc.hist[0].numpy(), floor=0.05) < 1e-3
    assert np.array_equal(tgn.embedding_module.histories[0].cache_flag != 0, orc.cache_flag[0] != 0)


def test_large_uncached_sets_take_the_bitmap_path():
    """Batches whose uncached set exceeds the candidate list (ORCA_CAND_CAP) fall back to the bitmap
    scan; both finishes must give the oracle's rows (counts, scores, pushed history rows)."""
    import dataclasses
    from orca_b200 import _lib, params, synthetic
    from oracle import tgn_oracle
    spec = dataclasses.replace(synthetic.SPECS["t_nb2"], name="wide", n_src=30000, n_edges=24000, budget=40, bs=1500,
                               zipf_src=0.3, zipf_dst=0.3)
    g = synthetic.make_graph(spec, seed=3)
    adj = tgn_oracle.Adjacency(g.sources, g.destinations, g.edge_idxs, g.timestamps, g.n_nodes)
    sd = params.random_state_dict(2, seed=4)
    orc = tgn_oracle.OracleTGN(adj, g.edge_features, sd, g.n_nodes, n_layers=2, budget=spec.budget)
    tgn = make_model(g)
    t = {k: torch.from_numpy(v) for k, v in sd.items()}
    t["embedding_module.time_encoder.w.weight"] = t["time_encoder.w.weight"]
    t["embedding_module.time_encoder.w.bias"] = t["time_encoder.w.bias"]
    tgn.load_state_dict(t)
    neg = synthetic.negative_destinations(g, seed=6)
    worst, sizes = 0.0, []
    for b, src, dst, ts, eidx in batches(g, 8):
        ng = neg[b * spec.bs: b * spec.bs + len(src)]
        pl = np.zeros(0, dtype=np.int64)     # empty plan: nothing stays cached
        rec = []
        wp, wq = orc.compute_edge_probabilities(src, dst, ng, ts, eidx, spec.n_degree, pl, record=rec)
        p, q = tgn.compute_edge_probabilities(src, dst, ng, ts, eidx, spec.n_degree, True, False, pl)
        n1, _, _ = tgn.check_status()
        assert n1 == 3 * len(src) + len(rec[0]), f"batch {b}"
        sizes.append(len(rec[0]))
        worst = max(worst, max_rel(p.cpu().numpy(), wp.numpy()), max_rel(q.cpu().numpy(), wq.numpy()))
    assert min(sizes[1:]) < _lib.CAND_CAP < max(sizes), sizes     # both finishes were exercised
    assert worst < 1e-3, worst
    assert max_rel(tgn.embedding_module.histories[0].emb.cpu().numpy(), orc.hist[0].numpy(), floor=0.05) < 1e-3


@pytest.mark.parametrize("case,reuse", [("t_nb2_reuse0", True), ("t_nb2_noreuse", False)])
def test_other_recursions_match_reference_fixture(case, reuse):
    """compute_embedding_reuse (budget == 0) and compute_embedding (reuse=False) of the reference,
    modules/embedding_module.py:154-182 and :116-147."""
    gold = golden(case)
    g = graph(str(gold["spec"]))
    spec = g.spec
    scores, neg = gold["scores"], gold["neg"]
    tgn = make_model(g, reuse=reuse, budget=0)
    worst = 0.0
    for b, src, dst, ts, eidx in batches(g, scores.shape[0]):
        n = len(src)
        p, q = tgn.compute_edge_probabilities(src, dst, neg[b * spec.bs: b * spec.bs + n], ts, eidx,
                                              spec.n_degree, reuse, False, None)
        n1, n_pos, _ = tgn.check_status()
        assert n1 == (3 * n if reuse else 3 * n * (1 + spec.n_degree))
        assert n_pos == len(np.unique(np.r_[src, dst]))
        worst = max(worst, max_rel(p.cpu().numpy().ravel(), scores[b, 0, :n]),
                    max_rel(q.cpu().numpy().ravel(), scores[b, 1, :n]))
    assert worst < 1e-3, worst
    pick = gold["state_nodes"].astype(np.int64)
    assert max_rel(tgn.memory.memory[pick].cpu().numpy(), gold["state_memory"], floor=0.05) < 1e-3
    if reuse:
        h = tgn.embedding_module.histories[0]
        assert max_rel(h.emb[pick].cpu().numpy(), gold["state_history"], floor=0.05) < 1e-3


def test_recursions_share_one_model():
    """The call's `reuse` argument picks the recursion per batch (model/tgn_model.py:114-120): a model
    built with history tables also serves reuse=False, and gives the scores of a model without."""
    g = graph("t_nb2")
    a, b = make_model(g, reuse=True), make_model(g, reuse=False, budget=0)
    spec = g.spec
    for i, src, dst, ts, eidx in batches(g, 3):
        neg = np.roll(dst, 1)
        pa, qa = a.compute_edge_probabilities(src, dst, neg, ts, eidx, spec.n_degree, False, False, None)
        pb, qb = b.compute_edge_probabilities(src, dst, neg, ts, eidx, spec.n_degree, False, False, None)
        a.check_status(), b.check_status()
        assert torch.equal(pa, pb) and torch.equal(qa, qb)
    with pytest.raises(AttributeError):
        b.compute_edge_probabilities(src, dst, neg, ts, eidx, spec.n_degree, True, False, None)


@pytest.mark.parametrize("option", ["dependent_launch", "lookahead", "overlap"])
def test_scheduling_switches_change_nothing(option):
    """Programmatic dependent launch, the four-stream look-ahead of the batch pipeline and the side stream
    of the raw-message / GRU chain only change WHEN kernels run: scores and state tables must be bit-identical
    with each of them off."""
    from orca_b200 import _lib
    g = graph("t_nb2")
    spec = g.spec
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    opt = {"dependent_launch": _lib.OPT_DEPENDENT_LAUNCH, "lookahead": _lib.OPT_LOOKAHEAD,
           "overlap": _lib.OPT_OVERLAP}[option]
    out = []
    for enable in (0, 1):
        tgn = make_model(g)
        tgn.set_option(opt, enable)
        scores = []
        for b, src, dst, ts, eidx in batches(g, 12):
            # no synchronisation between the batches: the lanes really run ahead of each other
            p, q = tgn.compute_edge_probabilities(src, dst, np.roll(dst, 1), ts, eidx, spec.n_degree, True, False,
                                                  plan[b])
            scores.append(torch.cat([p, q]))
        tgn.check_status()
        out.append((torch.cat(scores).clone(), tgn.memory.memory.clone(), tgn.memory.messages.clone(),
                    tgn.embedding_module.histories[0].emb.clone(),
                    tgn.embedding_module.histories[0].cache_flag_dev.clone()))
    for a, b in zip(out[0], out[1]):
        assert torch.equal(a, b)


def test_batches_of_changing_size_share_a_model():
    """A stream whose batches differ in size (the short last batch of every stream) lays the workspace out
    anew while the previous batch may still be in flight on the library's side streams."""
    g = graph("t_nb2")
    spec = g.spec
    sizes = [200, 37, 200, 5, 163, 200]
    ref, tgn = make_model(g), make_model(g)
    from orca_b200 import _lib
    ref.set_option(_lib.OPT_LOOKAHEAD, 0)
    lo = 0
    got, want = [], []
    for n in sizes:
        sl = slice(lo, lo + n)
        a = (g.sources[sl], g.destinations[sl], np.roll(g.destinations[sl], 1), g.timestamps[sl], g.edge_idxs[sl])
        plan = np.unique(np.r_[a[0], a[1]])[: spec.budget]
        want.append(torch.cat(ref.compute_edge_probabilities(*a, spec.n_degree, True, False, plan)))
        ref.check_status()        # the reference run is synchronised batch by batch, this one is not
        got.append(torch.cat(tgn.compute_edge_probabilities(*a, spec.n_degree, True, False, plan)))
        lo += n
    tgn.check_status()
    assert torch.equal(torch.cat(got), torch.cat(want))
    assert torch.equal(tgn.memory.memory, ref.memory.memory)
    assert torch.equal(tgn.embedding_module.histories[0].emb, ref.embedding_module.histories[0].emb)


@pytest.mark.parametrize("case", ["t_nb2", "t_lru"])
def test_eval_epoch_equals_per_batch_calls(case):
    """One library call for the whole stream (TGN.eval_epoch) gives the bits of one
    compute_edge_probabilities call per batch: scores and every state table; the stream's last batch is
    short, a few batches run without a plan."""
    gold = golden(case)
    g = graph(str(gold["spec"]))
    spec = g.spec
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    neg = gold["neg"]
    E = (len(plan) - 1) * spec.bs - 37           # a short last batch
    nb = -(-E // spec.bs)
    a, b = make_model(g), make_model(g)
    pos, ngs = [], []
    for i in range(nb):
        sl = slice(i * spec.bs, min(E, (i + 1) * spec.bs))
        p, q = a.compute_edge_probabilities(g.sources[sl], g.destinations[sl], neg[sl], g.timestamps[sl],
                                            g.edge_idxs[sl], spec.n_degree, True, False, plan[i])
        pos.append(p.cpu().numpy().ravel()), ngs.append(q.cpu().numpy().ravel())
    a.check_status()
    p2, q2 = b.eval_epoch(g.sources[:E], g.destinations[:E], neg[:E], g.timestamps[:E], g.edge_idxs[:E],
                          spec.n_degree, spec.bs, plan[:nb])
    b.check_status()
    assert np.array_equal(np.concatenate(pos), p2) and np.array_equal(np.concatenate(ngs), q2)
    assert torch.equal(a.memory.memory, b.memory.memory) and torch.equal(a.memory.messages, b.memory.messages)
    assert torch.equal(a.embedding_module.histories[0].emb, b.embedding_module.histories[0].emb)
    assert torch.equal(a.embedding_module.histories[0].cache_flag_dev, b.embedding_module.histories[0].cache_flag_dev)
    # a second epoch on the same model (staging ring and pinned buffers reused), without plans
    p3, _ = b.eval_epoch(g.sources[:E], g.destinations[:E], neg[:E], g.timestamps[:E], g.edge_idxs[:E],
                         spec.n_degree, spec.bs, None)
    b.check_status()
    assert p3.shape == (E,) and np.all((p3 > 0) & (p3 < 1))


def test_eval_edge_prediction_reproduces_reference_ap():
    """The reference's evaluation entry point (evaluation/evaluation.py:6-47) on the whole c1 stream: the
    mean average precision of the fixture the reference produced, to 3 decimals."""
    import types
    from orca_b200.evaluation import RandEdgeSampler, eval_edge_prediction
    gold = golden("c1")
    g = graph(str(gold["spec"]))
    spec = g.spec
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    nb = gold["scores"].shape[0]
    n = min(g.n_edges, nb * spec.bs)
    data = types.SimpleNamespace(sources=g.sources, destinations=g.destinations, timestamps=g.timestamps,
                                 edge_idxs=g.edge_idxs, n_interactions=n)
    sampler = RandEdgeSampler(g.sources, g.destinations, seed=0)
    tgn = make_model(g)
    ap, auc, acc = eval_edge_prediction(tgn, sampler, data, spec.n_degree, spec.bs, True, plan)
    tgn.check_status()
    assert round(float(ap), 3) == round(float(gold["ap"]), 3)
    assert 0.0 <= auc <= 1.0 and 0.0 <= acc <= 1.0


def test_unsupported_modes_fail_loudly():
    g = graph("t_nb2")
    tgn = make_model(g)
    src, dst, ts, eidx = g.sources[:10], g.destinations[:10], g.timestamps[:10], g.edge_idxs[:10]
    with pytest.raises(NotImplementedError):
        tgn.compute_edge_probabilities(src, dst, dst, ts, eidx, 10, True, True, None)


@pytest.mark.parametrize("world,direct", [(4, False), (8, False), (2, True), (8, True), (3, "split"), (2, "layers"),
                                          (5, "layers"), (8, "layers")])
def test_sharded_entry_points_with_emulated_ranks(world, direct):
    """The row/edge split of the multi-GPU path for more ranks than GPUs at hand: every rank is a model
    replica of its own on this GPU, the two phases are called rank after rank through the C ABI (all ranks'
    phase 1 before any phase 2, so no kernel ever waits for a later launch).  The exchange between the
    phases is a stack of the ranks' layer-1 rows, or -- direct -- the library's own peer stores into every
    replica's exchange buffer.  "split": the memory update is split by node too; "layers": the first half of
    the ranks computes layer 1 and the memory update, the second half the top layer and the scores.  Scores
    and state must equal the unsharded run."""
    from orca_b200 import _lib, shard
    L = _lib.lib()
    g = graph("t_nb2")
    spec = g.spec
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    ref = make_model(g)
    ranks = [make_model(g) for _ in range(world)]
    for r, m in enumerate(ranks):
        m._rank, m._world = r, world
        # one stream for everything: the ranks share this GPU, and a rank's wait for its peers' rows must
        # never be scheduled ahead of the kernels that deliver them
        m.set_option(_lib.OPT_LOOKAHEAD, 0)
        m.set_option(_lib.OPT_OVERLAP, 0)
    dev = ref.device
    if direct:
        # the ranks' exchange buffers and flag words; on one GPU a "peer" address is a plain device address
        from orca_b200.tgn import TGN
        cap = TGN.exchange_floats(spec.bs, world, spec.n_degree, g.n_nodes)
        bufs = [torch.zeros(_lib.EXCHANGE_SLOTS * cap, device=dev) for _ in range(world)]
        flags = [torch.zeros(_lib.FLAG_WORDS, dtype=torch.int32, device=dev) for _ in range(world)]
        # "split": the memory update is split by node as well, its rows exchanged the same way
        gcap = 2 * spec.bs * 172
        grus = [torch.zeros(2 * gcap, device=dev) for _ in range(world)] if direct in ("split", "layers") else None
        for m in ranks:
            m.set_exchange([x.data_ptr() for x in bufs], [f.data_ptr() for f in flags], cap, bufs + flags,
                           [x.data_ptr() for x in grus] if grus else None, gcap)
            m._keep_gru = grus
            if direct == "layers":
                m._layer1_ranks = world // 2
    wa = world // 2 if direct == "layers" else 0        # ranks wa.. hold the scores
    wb = world - wa
    stream = _lib.stream_ptr(dev)
    k = spec.n_degree
    worst = 0.0
    for b, src, dst, ts, eidx in batches(g, 8):
        n = len(src)
        neg = np.roll(dst, 3)
        p_ref, q_ref = ref.compute_edge_probabilities(src, dst, neg, ts, eidx, k, True, False, plan[b])
        ref.check_status()
        pl = np.asarray(plan[b], dtype=np.int32)
        ints = torch.from_numpy(np.concatenate([src, dst, neg, eidx, pl]).astype(np.int32)).to(dev)
        tsd = torch.from_numpy(np.ascontiguousarray(ts, dtype=np.float64)).to(dev)
        d_plan = ints.data_ptr() + 16 * n
        locals_, ctx = [], []
        for m in ranks:
            desc = m._descriptor(k)
            ws, u_cap = m._workspace(n, k)
            rpr = shard.rows_per_rank(3 * n + u_cap, wa if wa else world)
            emb1 = torch.zeros(rpr, 172, device=dev)
            _lib.check(L.orca_tgn_eval_batch_sharded(desc, 1, ints.data_ptr(), tsd.data_ptr(), n, d_plan, len(pl),
                                                     u_cap, ws.data_ptr(), ws.numel(),
                                                     None if direct else emb1.data_ptr(), None, None,
                                                     None, m._status.data_ptr(), stream))
            locals_.append(emb1)
            ctx.append((desc, ws, u_cap))
        emb1_all = torch.stack(locals_).contiguous()
        p = torch.zeros(n, device=dev)
        q = torch.zeros(n, device=dev)
        for r, m in enumerate(ranks):
            desc, ws, u_cap = ctx[r]
            n_loc = shard.local_count(n, r - wa, wb) if r >= wa else 0
            prob = torch.zeros(2 * shard.rows_per_rank(n, wb), device=dev)
            _lib.check(L.orca_tgn_eval_batch_sharded(desc, 2, ints.data_ptr(), tsd.data_ptr(), n, d_plan, len(pl),
                                                     u_cap, ws.data_ptr(), ws.numel(), None,
                                                     None if direct else emb1_all.data_ptr(),
                                                     prob.data_ptr(), None, m._status.data_ptr(), stream))
            m.check_status()
            if r >= wa:
                e = torch.arange(r - wa, n, wb, device=dev)
                p[e] = prob[:n_loc]
                q[e] = prob[n_loc:2 * n_loc]
        worst = max(worst, float((p - p_ref.view(-1)).abs().max()), float((q - q_ref.view(-1)).abs().max()))
    assert worst < 1e-6, worst
    for m in ranks:
        assert torch.equal(m.memory.memory, ref.memory.memory)
        assert torch.equal(m.embedding_module.histories[0].emb, ref.embedding_module.histories[0].emb)
        assert np.array_equal(m.embedding_module.histories[0].cache_flag, ref.embedding_module.histories[0].cache_flag)


def test_wait_for_peers_gives_up_and_leaves_the_tables_alone():
    """A rank whose peer never delivers its rows: the bounded waits of phase 2 run out (the limit is set to
    about a millisecond), the status word reports ORCA_E_TIMEOUT, the kernels return, and neither the history
    replica nor the memory table receives rows from the incomplete exchange.  Nothing faults or hangs: the
    wait is a poll of a flag word that is never set."""
    from orca_b200 import _lib, shard
    from orca_b200.tgn import TGN
    L = _lib.lib()
    g = graph("t_nb2")
    spec = g.spec
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    world = 2
    m = make_model(g)
    m._rank, m._world = 0, world
    m.set_option(_lib.OPT_LOOKAHEAD, 0)
    m.set_option(_lib.OPT_OVERLAP, 0)
    m.set_option(_lib.OPT_WAIT_LIMIT, 2_000_000)
    dev = m.device
    cap = TGN.exchange_floats(spec.bs, world, spec.n_degree, g.n_nodes)
    gcap = 2 * spec.bs * 172
    bufs = [torch.zeros(_lib.EXCHANGE_SLOTS * cap, device=dev) for _ in range(world)]
    flags = [torch.zeros(_lib.FLAG_WORDS, dtype=torch.int32, device=dev) for _ in range(world)]
    grus = [torch.zeros(2 * gcap, device=dev) for _ in range(world)]
    m.set_exchange([x.data_ptr() for x in bufs], [f.data_ptr() for f in flags], cap, bufs + flags + grus,
                   [x.data_ptr() for x in grus], gcap)
    _, src, dst, ts, eidx = next(iter(batches(g, 1)))
    n, k = len(src), spec.n_degree
    pl = np.asarray(plan[0], dtype=np.int32)
    ints = torch.from_numpy(np.concatenate([src, dst, np.roll(dst, 3), eidx, pl]).astype(np.int32)).to(dev)
    tsd = torch.from_numpy(np.ascontiguousarray(ts, dtype=np.float64)).to(dev)
    desc = m._descriptor(k)
    ws, u_cap = m._workspace(n, k)
    hist_before = m.embedding_module.histories[0].emb.clone()
    mem_before = m.memory.memory.clone()
    prob = torch.zeros(2 * shard.rows_per_rank(n, world), device=dev)
    stream = _lib.stream_ptr(dev)
    for phase in (1, 2):        # rank 1 never runs: its flag words stay zero
        _lib.check(L.orca_tgn_eval_batch_sharded(desc, phase, ints.data_ptr(), tsd.data_ptr(), n,
                                                 ints.data_ptr() + 16 * n, len(pl), u_cap, ws.data_ptr(), ws.numel(),
                                                 None, None, prob.data_ptr(), None, m._status.data_ptr(), stream))
    with pytest.raises(_lib.OrcaError) as err:
        m.check_status()
    assert err.value.code == 6          # ORCA_E_TIMEOUT
    assert torch.equal(m.embedding_module.histories[0].emb, hist_before)
    assert torch.equal(m.memory.memory, mem_before)
    # the context is still usable: an unsharded model on the same GPU runs a batch
    ok = make_model(g)
    p, q = ok.compute_edge_probabilities(src, dst, np.roll(dst, 3), ts, eidx, k, True, False, plan[0])
    ok.check_status()
    assert torch.isfinite(p).all() and torch.isfinite(q).all()


def test_device_side_errors_surface_through_the_reference_api():
    """The reference API has no status call.  What a kernel reports in the status word (here: the code a kernel
    writes when the uncached set exceeds its capacity, put there by the host so that no kernel has to fail)
    travels to pinned host memory behind each batch and is raised by the first later call that finds the copy
    complete."""
    from orca_b200 import _lib
    g = graph("t_nb2")
    spec = g.spec
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    m = make_model(g)
    it = iter(batches(g, 3))
    _, src, dst, ts, eidx = next(it)
    m.compute_edge_probabilities(src, dst, np.roll(dst, 3), ts, eidx, spec.n_degree, True, False, plan[0])
    torch.cuda.synchronize()
    m._status[0] = 4                     # ORCA_E_CAPACITY, as report() would leave it
    _, src, dst, ts, eidx = next(it)
    m.compute_edge_probabilities(src, dst, np.roll(dst, 3), ts, eidx, spec.n_degree, True, False, plan[1])
    torch.cuda.synchronize()
    _, src, dst, ts, eidx = next(it)
    with pytest.raises(_lib.OrcaError) as err:
        m.compute_edge_probabilities(src, dst, np.roll(dst, 3), ts, eidx, spec.n_degree, True, False, plan[2])
    assert err.value.code == 4


@pytest.mark.parametrize("planned", [True, False])      # groups of batches / batch by batch
def test_device_side_errors_of_a_stream_are_raised_by_its_own_call(planned):
    """A user who scores a stream in one call has no later call to hear of an error through: eval_epoch raises what
    its kernels left in the status word (here put there by the host), once, and the next stream runs."""
    from orca_b200 import _lib
    g = graph("t_nb2")
    spec = g.spec
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"]) if planned else None
    m = make_model(g)
    E = 3 * spec.bs
    run = lambda: m.eval_epoch(g.sources[:E], g.destinations[:E], np.roll(g.destinations[:E], 3), g.timestamps[:E],
                               g.edge_idxs[:E], spec.n_degree, spec.bs, plan)
    run()
    m._status[0] = 6                     # ORCA_E_TIMEOUT, as report() would leave it
    with pytest.raises(_lib.OrcaError) as err:
        run()
    assert err.value.code == 6
    pos, neg = run()
    assert np.isfinite(pos).all() and np.isfinite(neg).all()


@pytest.mark.parametrize("layers", [1, 2])
def test_an_id_outside_its_table_is_refused(layers):
    """A node or edge id that the tables have no row for, in each array of a batch, first and last entry, is an error of
    the call.  A batch of a single call has never been there (its kernels would read the rows of its ids unchecked); the
    kernels of a group guard theirs."""
    import dataclasses
    from orca_b200 import _lib
    g = graph("t_nb2")
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, n_layers=layers))
    spec = g.spec
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    E, k, bs = 2 * spec.bs + 5, spec.n_degree, spec.bs
    good = [g.sources[:E], g.destinations[:E], np.roll(g.destinations[:E], 3), g.timestamps[:E], g.edge_idxs[:E]]
    m, other = make_model(g), make_model(g)
    call = lambda m, x, i: m.compute_edge_probabilities(*[a[i * bs:(i + 1) * bs] for a in x], k, True, False, plan[i])
    call(m, good, 0), call(other, good, 0)
    for which, lim in ((0, g.n_nodes), (1, g.n_nodes), (2, g.n_nodes), (4, g.n_edges + 1)):
        for at, bad in ((bs, -1), (2 * bs - 1, lim), (bs + 3, 1 << 32)):
            x = [np.array(a) for a in good]
            x[which][at] = bad
            with pytest.raises(_lib.OrcaError) as err:
                call(m, x, 1)
            assert err.value.code == 5           # ORCA_E_BOUNDS
            if bad == 1 << 32:                   # (a stream's arrays are narrowed by numpy)
                continue
            for p in (plan, None):
                with pytest.raises(_lib.OrcaError) as err:
                    make_model(g).eval_epoch(*x, k, bs, p)
                assert err.value.code == 5
    for a, b in zip(call(m, good, 1), call(other, good, 1)):
        assert torch.equal(a, b)
    assert torch.equal(m.memory.memory, other.memory.memory)


def test_the_status_copy_serves_every_path_whichever_ran_first():
    """The calls of one GPU, whole streams and the batches of the multi-GPU split share the pinned status word: a model
    that has scored on its own can be split afterwards (the end of a split batch is called by hand here)."""
    from orca_b200 import _lib
    g = graph("t_nb2")
    spec = g.spec
    for first in ("call", "stream"):
        m = make_model(g)
        _, src, dst, ts, eidx = next(iter(batches(g, 1)))
        batch = (src, dst, np.roll(dst, 3), ts, eidx)
        if first == "call":
            m.compute_edge_probabilities(*batch, spec.n_degree, True, False, None)
        else:
            m.eval_epoch(*batch, spec.n_degree, spec.bs, None)
        m.check_status()
        m._status[0] = 4                 # ORCA_E_CAPACITY, as report() would leave it
        m._ev_free = [None]
        m._release_dev(0, torch.cuda.current_stream())
        torch.cuda.synchronize()
        with pytest.raises(_lib.OrcaError) as err:
            m.compute_edge_probabilities(*batch, spec.n_degree, True, False, None)
        assert err.value.code == 4


def test_edge_features_can_be_replaced_between_calls():
    """``edge_raw_features`` is an attribute of the model, as in the reference: a table put in its place is the one
    that the next call reads (the old one is kept alive here)."""
    g = graph("t_nb2")
    spec = g.spec
    m, fresh = make_model(g), make_model(g)
    old = m.edge_raw_features
    table = torch.cat([old * -0.5 + 0.25, old])
    it = iter(batches(g, 2))
    for _, src, dst, ts, eidx in it:
        batch = (src, dst, np.roll(dst, 3), ts, eidx, spec.n_degree, True, False, None)
        a, b = m.compute_edge_probabilities(*batch), fresh.compute_edge_probabilities(*batch)
        if m.edge_raw_features is old:
            assert all(torch.equal(x, y) for x, y in zip(a, b))
            m.edge_raw_features = table
            fresh.edge_raw_features.copy_(table[:len(old)])
    assert all(torch.equal(x, y) for x, y in zip(a, b))


def _after_a_long_kernel(f):
    """f() behind some milliseconds of work on the caller's stream: what it enqueues there runs late."""
    torch.cuda._sleep(20_000_000)
    return f()


def test_a_batch_sees_what_was_written_on_the_callers_stream():
    """Tables replaced, written in place or written by the library's own calls between two batches, and weights that
    are packed at the first one, are complete when a batch starts on the library's streams; copies taken between two
    batches hold what the first one left."""
    g = graph("t_nb2")
    spec = g.spec
    k = spec.n_degree
    gold = golden("t_nb2")
    plan = unpack(gold[f"plan_{spec.strategy}_flat"], gold[f"plan_{spec.strategy}_off"])
    bat = [(s, d, np.roll(d, 3), t, e, k, True, False, plan[b]) for b, s, d, t, e in batches(g, 4)]

    def want(change):     # the same with everything waited for
        m = make_model(g)
        for i, x in enumerate(bat[:3]):
            if i == 2:
                change(m)
                torch.cuda.synchronize()
            r = m.compute_edge_probabilities(*x)
            torch.cuda.synchronize()
        return [t.cpu() for t in r] + [m.memory.memory.cpu()]

    rows = torch.randn(g.n_nodes, 172, device="cuda")
    ids = np.arange(1, g.n_nodes)
    shift = (torch.randn(g.n_nodes, device="cuda") * 5).cpu()
    state = make_model(g).memory.backup_memory()
    changes = [lambda m: m.memory.memory.copy_(rows),
               lambda m: m.memory.set_memory(ids, rows[1:]),
               lambda m: m.memory.restore_memory((rows,) + state[1:]),
               lambda m: m.embedding_module.histories[0].emb.copy_(rows),
               lambda m: m.embedding_module.histories[0].push(rows[1:], ids),
               lambda m: m.embedding_module.histories[0].update_flag(ids[::3], None),
               lambda m: m.embedding_module.reset_history(),
               lambda m: m.memory.last_update.copy_(shift.cuda()),
               lambda m: m.edge_raw_features.mul_(0.5)]
    for n, change in enumerate(changes):
        w = want(change)
        m = make_model(g)
        for x in bat[:2]:
            m.compute_edge_probabilities(*x)
        _after_a_long_kernel(lambda: change(m))
        r = [t.cpu() for t in m.compute_edge_probabilities(*bat[2])] + [m.memory.memory.cpu()]
        assert all(torch.equal(a, b) for a, b in zip(r, w)), n
    # weights packed late, at the first call
    w = want(lambda m: m.refresh_weights())
    m = make_model(g)
    for x in bat[:2]:
        m.compute_edge_probabilities(*x)
    m.refresh_weights()
    torch.cuda._sleep(20_000_000)
    r = [t.cpu() for t in m.compute_edge_probabilities(*bat[2])] + [m.memory.memory.cpu()]
    assert all(torch.equal(a, b) for a, b in zip(r, w))
    # copies taken between two batches
    m, o = make_model(g), make_model(g)
    for x in bat[:2]:
        m.compute_edge_probabilities(*x), o.compute_edge_probabilities(*x)
    torch.cuda.synchronize()
    late = _after_a_long_kernel(lambda: (*m.memory.backup_memory(), *m.embedding_module.backup_history(),
                                         m.memory.get_memory(ids), m.memory.get_last_update(ids),
                                         m.embedding_module.histories[0].pull(ids)))
    m.compute_edge_probabilities(*bat[2])
    now = (*o.memory.backup_memory(), *o.embedding_module.backup_history(), o.memory.get_memory(ids),
           o.memory.get_last_update(ids), o.embedding_module.histories[0].pull(ids))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(late, now))
    # a table that the caller reads itself, before a whole stream
    E = spec.bs
    for p in (plan[3:4], None):
        m = make_model(g)
        for x in bat[:2]:
            m.compute_edge_probabilities(*x)
        torch.cuda.synchronize()
        before = m.memory.memory.cpu()
        late = _after_a_long_kernel(lambda: m.memory.memory.clone())
        m.eval_epoch(g.sources[3 * E:4 * E], g.destinations[3 * E:4 * E], bat[3][2], g.timestamps[3 * E:4 * E],
                     g.edge_idxs[3 * E:4 * E], k, E, p)
        assert torch.equal(late.cpu(), before)


def test_a_model_made_in_inference_mode_scores():
    g = graph("t_nb2")
    with torch.inference_mode():
        m = make_model(g)
        _, s, d, t, e = next(iter(batches(g, 1)))
        out = [m.compute_edge_probabilities(s, d, np.roll(d, 3), t, e, g.spec.n_degree, True, False, None) for _ in range(2)]
    o = make_model(g)
    for r in out:
        for a, b in zip(r, o.compute_edge_probabilities(s, d, np.roll(d, 3), t, e, g.spec.n_degree, True, False, None)):
            assert torch.equal(a, b)


def test_a_call_takes_the_forms_of_arrays_it_took_before():
    """Lists, other types, strided arrays, one value for all, a matrix of one row: what plain arrays give.  Another
    length or a matrix with a row per edge is refused."""
    g = graph("t_nb2")
    k = g.spec.n_degree
    _, src, dst, ts, eidx = next(iter(batches(g, 1)))
    neg = np.full(len(src), dst[0])
    plan = np.arange(5, 50)
    run = lambda *a, plan=plan: [t.cpu() for t in make_model(g).compute_edge_probabilities(*a, k, True, False, plan)]
    want = run(src, dst, neg, ts, eidx)
    for a in ((list(src), list(dst), list(neg), list(ts), list(eidx)),
              (src.astype(np.int32), dst.astype(np.float64), neg, ts, np.repeat(eidx, 2)[::2]),
              (torch.from_numpy(np.array(src)), dst, dst[:1], ts, eidx),
              (src, dst, dst[0], ts, eidx),
              (src, dst[None, :], neg, ts[None, :], eidx)):
        assert all(torch.equal(x, y) for x, y in zip(run(*a, plan=list(plan)), want))
    for a in ((src, dst[:-1], neg, ts, eidx), (src, dst, np.r_[neg, 1], ts, eidx), (src, dst, neg, ts[:0], eidx),
              (src, dst, np.stack([neg, neg], 1), ts, eidx), (src, dst, neg, ts[:, None], eidx)):
        with pytest.raises(ValueError):
            run(*a)


@pytest.mark.parametrize("name,reuse,budget,updates", [("c1", True, None, True), ("t_nb2", True, None, True),
                                                       ("t_nb2", True, 0, False), ("t_nb2", False, None, False)])
def test_a_call_that_fails_half_way_leaves_nothing_in_flight(name, reuse, budget, updates):
    """A batch whose scorer is refused (no weights) has enqueued its layers and, in the first two recursions, on a stream of
    the library's own, its memory update by then.  All of it has finished when the error is raised, although it stood behind
    0.1 s of other work, and the model goes on."""
    from orca_b200 import _lib
    g = graph(name)
    k = g.spec.n_degree
    m = make_model(g, reuse=reuse, budget=budget)
    run = lambda i: m.compute_edge_probabilities(*[a[200 * i:200 * (i + 1)] for a in (
        g.sources, g.destinations, np.roll(g.destinations, 1), g.timestamps, g.edge_idxs)], k, reuse, False, None)
    run(0)
    m.check_status()
    before = m.memory.memory.clone()
    torch.cuda.synchronize()
    weights, m._desc.score.W1t = m._desc.score.W1t, None
    torch.cuda._sleep(200_000_000)
    with pytest.raises(_lib.OrcaError):
        run(1)
    assert torch.cuda.current_stream().query()
    beside = torch.cuda.Stream()
    with torch.cuda.stream(beside):
        now = m.memory.memory.clone()
    torch.cuda.synchronize()
    assert torch.equal(now, m.memory.memory) and torch.equal(now, before) != updates
    m._desc.score.W1t = weights
    pos, neg = run(2)
    m.check_status()
    assert torch.isfinite(pos).all() and torch.isfinite(neg).all()


@pytest.mark.parametrize("option", ["dependent_launch", "overlap"])
@pytest.mark.parametrize("name,reuse,budget", [("c1", True, None), ("t_nb2", True, 0), ("t_nb2", False, None)])
def test_switches_change_nothing_in_the_recursions_on_two_streams(name, reuse, budget, option):
    """One layer, unlimited reuse and no reuse: the memory update runs on a stream of its own beside a layer.  Calls of
    changing size, back to back without a synchronisation, give the same bits with it off."""
    from orca_b200 import _lib
    g = graph(name)
    k = g.spec.n_degree
    opt = {"dependent_launch": _lib.OPT_DEPENDENT_LAUNCH, "overlap": _lib.OPT_OVERLAP}[option]
    sizes = [37, 200, 5, 130, 1100, 64, 37, 1] * 2      # (more than 1024 edges: the update as a pair of launches)
    out = []
    for enable in (0, 1):
        m = make_model(g, reuse=reuse, budget=budget)
        m.set_option(opt, enable)
        scores, lo = [], 0
        for n in sizes:
            a = [x[lo:lo + n] for x in (g.sources, g.destinations, np.roll(g.destinations, 1), g.timestamps, g.edge_idxs)]
            scores += m.compute_edge_probabilities(*a, k, reuse, False, None)
            lo += n
        m.check_status()
        out.append([torch.cat(scores)] + [getattr(m.memory, t).clone() for t in ("memory", "last_update", "messages",
                                                                                 "timestamps", "nodes_dev")])
    assert lo <= g.n_edges
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("projection", [0, 1])
@pytest.mark.parametrize("name", ["c1", "t_nb2"])
def test_values_that_are_not_numbers_reach_the_scores(name, projection):
    """A node whose memory is not a number: in the first batch the scores of its own edges and of those that see it as a
    neighbour are NaN, as the reference's are, and the others are what they were."""
    from orca_b200 import _lib
    g = graph(name)
    k = g.spec.n_degree
    lo = g.n_edges // 2
    a = [x[lo:lo + 200] for x in (g.sources, g.destinations, np.roll(g.destinations, 1), g.timestamps, g.edge_idxs)]
    out = []
    for bad in (0.0, float("nan")):
        m = make_model(g)
        m.set_option(_lib.OPT_PROJECTION_MODE, projection)
        node = int(a[0][17])
        m.memory.memory[node] = bad
        out.append([t.cpu().numpy().ravel() for t in m.compute_edge_probabilities(*a, k, False, False, None)])
        m.check_status()
    own = a[0] == node
    for score, was, ends in zip(out[1], out[0], (own | (a[1] == node), own | (a[2] == node))):
        assert np.isnan(score[ends]).all()
        assert np.isfinite(was).all() and np.isfinite(score).any()
        assert np.array_equal(score[~np.isnan(score)], was[~np.isnan(score)])


@pytest.mark.parametrize("layers", [1, 2])
def test_a_graph_that_knows_fewer_nodes_than_the_model(layers):
    """get_neighbor_finder(data) knows nodes up to the largest id of its edges.  Edges of nodes beyond that are scored as
    those of nodes without interactions: the same bits as with a graph that has empty lists for them."""
    import dataclasses
    import types
    from orca_b200.neighbor_finder import get_neighbor_finder
    g = graph("t_nb2")
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, n_layers=layers))
    k, low = g.spec.n_degree, g.n_nodes // 2
    pick = np.nonzero((g.sources < low) & (g.destinations < low))[0]
    part = types.SimpleNamespace(sources=g.sources[pick], destinations=g.destinations[pick], edge_idxs=g.edge_idxs[pick],
                                 timestamps=g.timestamps[pick])
    small, padded = get_neighbor_finder(part), get_neighbor_finder(part, max_node_idx=g.n_nodes - 1)
    assert small.n_nodes <= low < padded.n_nodes == g.n_nodes and (g.sources[-400:] >= low).any()
    a = [x[-400:] for x in (g.sources, g.destinations, np.roll(g.destinations, 1), g.timestamps, g.edge_idxs)]
    out = []
    for nf in (small, padded):
        m = make_model(g)
        m.set_neighbor_finder(nf)
        got = [np.r_[tuple(t.cpu().numpy().ravel() for t in m.compute_edge_probabilities(*[x[:200] for x in a], k, True, False,
                                                                                          None))]]
        got += m.eval_epoch(*a, k, 200, [np.zeros(0, np.int64)] * 2)
        m.check_status()
        out.append(got)
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("k", [10, 20])
@pytest.mark.parametrize("name,reuse,budget", [("c1", True, None), ("t_nb2", True, None), ("t_nb2", True, 0), ("t_nb2", False, None)])
def test_sampled_ids_without_rows_are_reported(name, reuse, budget, k):
    """A graph can name nodes or edges that the model's tables have no rows for.  A slot that one of them is sampled into is
    left empty and reported -- by a single call to a later one, by a stream when it ends -- and one that no query reaches
    does no harm."""
    import dataclasses
    from orca_b200 import _lib
    from orca_b200.neighbor_finder import NeighborFinder
    g = graph(name)
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, n_degree=k))
    hub = int(np.bincount(g.sources[:200]).argmax())
    a = [x[:200] for x in (g.sources, g.destinations, np.roll(g.destinations, 1), g.timestamps, g.edge_idxs)]
    a[3] = a[3] + 10.0

    def lists(node, edge, time):
        own = [np.zeros(0)] * g.n_nodes
        own[hub] = np.array([1, node, 2])
        return NeighborFinder(own, [np.array([3, edge, 4])[:len(x)] for x in own], [np.array([1.0, time, time])[:len(x)] for x in own])

    def run(nf, stream):
        m = make_model(g, reuse=reuse, budget=budget)
        m.set_neighbor_finder(nf)
        plan = [np.zeros(0, np.int64)] * 4 if reuse and budget is None else None
        if stream:
            return m.eval_epoch(*a, k, 50, plan, reuse=reuse)
        s = m.compute_edge_probabilities(*a, k, reuse, False, plan[0] if plan else None)
        m.check_status()
        return [x.cpu().numpy() for x in s]
    for stream in (False, True):
        for node, edge in ((g.n_nodes, 1), (-1, 1), (2, g.n_edges + 1), (2, -5), (2 ** 31 - 1, 2 ** 31 - 1)):
            with pytest.raises(_lib.OrcaError) as e:
                run(lists(node, edge, 2.0), stream)
            assert e.value.code == _lib.E_BOUNDS
        late = run(lists(g.n_nodes, -5, 1e30), stream)      # (behind every query)
        for x, y in zip(run(lists(g.n_nodes - 1, g.n_edges, 1e30), stream), late):
            assert np.array_equal(x, y) and np.isfinite(x).all()
        run(lists(g.n_nodes - 1, g.n_edges, 2.0), stream)


@pytest.mark.parametrize("b", [1, 63, 64, 65, 128, 200, 1100])
def test_updates_of_a_batch_against_64_bits(b):
    """Memory rows of a budgeted batch, whose messages come to the GRU as an operand image, against the GRU in 64 bits from the
    message table: fewer rows than a block, a block and a bit, several.  Operands carry 16 significant bits (relative error
    2^-17 each, both sides of a product): a gate's sum is off by 2^-16 of the sum of the products' sizes, the gates' slopes are
    at most 1/4 (twice) and 1, and the candidate is scaled by the reset gate's sum once more."""
    g = graph("c1")
    tgn = _two_layer_model(g, b)
    rs = np.random.RandomState(b)
    old = torch.from_numpy((rs.randn(g.n_nodes, 172) * 0.4).astype(np.float32)).cuda()
    tgn.memory.memory.copy_(old)
    lo = len(g.sources) // 2
    part = [x[lo:lo + b] for x in (g.sources, g.destinations, g.destinations[::-1], g.timestamps, g.edge_idxs)]
    tgn.compute_edge_probabilities(*part, 10, True, False, np.unique(part[0])[:20])
    tgn.check_status()
    nodes = np.unique(np.concatenate(part[:2]))
    p = "memory_updater.memory_updater."
    wi, wh, bi, bh = (torch.from_numpy(state_dict(2)[p + n]).double() for n in ("weight_ih", "weight_hh", "bias_ih", "bias_hh"))
    x, h = tgn.memory.messages.cpu()[nodes].double(), old.cpu()[nodes].double()
    assert torch.equal(x[:, :172].float(), old.cpu()[nodes])
    i, j = (x @ wi.T + bi).chunk(3, 1), (h @ wh.T + bh).chunk(3, 1)
    r, z = torch.sigmoid(i[0] + j[0]), torch.sigmoid(i[1] + j[1])
    want = (1 - z) * torch.tanh(i[2] + r * j[2]) + z * h
    size = (x.abs() @ wi.abs().T).chunk(3, 1), (h.abs() @ wh.abs().T).chunk(3, 1)
    off = [2.0 ** -16 * (a + c) for a, c in zip(*size)]
    bound = off[2] + off[0] / 4 * (1 + j[2].abs()) + off[1] / 4 * (1 + h.abs()) + 2e-6
    got = tgn.memory.memory.cpu().double()
    assert bool(((got[nodes] - want).abs() < bound).all())
    rest = np.setdiff1d(np.arange(g.n_nodes), nodes)
    assert torch.equal(got[rest].float(), old.cpu()[rest])


def _two_layer_model(g, bs):
    import dataclasses
    return make_model(dataclasses.replace(g, spec=dataclasses.replace(g.spec, bs=bs, n_layers=2, n_degree=10, budget=20)))


@pytest.mark.parametrize("layers", [1, 2])
@pytest.mark.parametrize("b", [1, 63, 64, 65, 128, 129, 300])
def test_scores_of_a_batch_are_those_of_its_embeddings(layers, b):
    """The pairs' operand image that the top layer leaves for the scorer, at its blocks' edges: the scores of a batch are bit
    for bit orca_score's of the embeddings that the same batch returns on a second model."""
    import dataclasses
    from orca_b200 import _lib
    g = graph("c1")
    g = dataclasses.replace(g, spec=dataclasses.replace(g.spec, bs=b, n_layers=layers, n_degree=10, budget=20))
    a, e = make_model(g), make_model(g)
    lo = len(g.sources) // 2
    part = [x[lo:lo + b] for x in (g.sources, g.destinations, np.roll(g.destinations, 7), g.timestamps, g.edge_idxs)]
    plan = np.unique(part[0])[:20] if layers == 2 else None
    pos, neg = a.compute_edge_probabilities(*part, 10, True, False, plan)
    emb = torch.cat(e.compute_temporal_embeddings(*part, 10, True, False, plan)).contiguous()
    want = torch.empty(2 * b, device=emb.device)
    _lib.check(_lib.lib().orca_score(e.score_struct(), emb.data_ptr(), b, want.data_ptr(), _lib.stream_ptr(emb.device)))
    a.check_status(), e.check_status()
    assert torch.equal(torch.cat([pos, neg]).ravel(), want)
