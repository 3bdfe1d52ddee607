"""Entry points that take host arrays at the edges of their chunks and tiles: the adjacency (chunks of 65 536 edges,
tiles of 8192 records, one to three bytes of node id, streams in and out of time order) from host and from device
arrays, and the neighbour tables."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _stream(E, n, sorted_ts, seed):
    rs = np.random.RandomState(seed)
    src, dst = rs.randint(0, n, E).astype(np.int64), rs.randint(0, max(1, n // 2), E).astype(np.int64)
    ts = np.round(rs.rand(E) * max(E // 3, 1))
    return src, dst, np.arange(1, E + 1, dtype=np.int64), np.sort(ts) if sorted_ts else ts


@pytest.mark.parametrize("E,n", [(0, 5), (1, 1), (4095, 256), (4096, 257), (4097, 70000), (65536, 65536), (65537, 65537),
                                 (300001, 1 << 20)])
@pytest.mark.parametrize("sorted_ts", [True, False])
def test_adjacency_from_host_and_device_arrays(E, n, sorted_ts):
    from oracle import tgn_oracle
    from orca_b200 import _lib
    from orca_b200.neighbor_finder import NeighborFinder
    src, dst, eidx, ts = _stream(E, n, sorted_ts, E + n)
    adj = tgn_oracle.Adjacency(src, dst, eidx, ts, n)
    nf = NeighborFinder.build_on_device(src, dst, eidx, ts, n)
    L = _lib.lib()
    dev = [torch.from_numpy(a).cuda() for a in (src, dst, eidx, ts)]
    indptr = torch.empty(n + 1, dtype=torch.int64, device="cuda")
    nbr, eid = (torch.empty(2 * E + 1, dtype=torch.int32, device="cuda") for _ in range(2))
    ats = torch.empty(2 * E + 1, dtype=torch.float64, device="cuda")
    ws = torch.empty(L.orca_csr_build_workspace_bytes(E, n), dtype=torch.uint8, device="cuda")
    status = torch.zeros(4, dtype=torch.int32, device="cuda")
    _lib.check(L.orca_csr_build(*(t.data_ptr() for t in dev), E, n, indptr.data_ptr(), nbr.data_ptr(), eid.data_ptr(),
                                ats.data_ptr(), status.data_ptr(), ws.data_ptr(), ws.numel(), _lib.stream_ptr()))
    assert status.cpu().tolist() == [0, 0, 0, 0]
    for got in ((nf.indptr, nf.adj_nbr, nf.adj_eid, nf.adj_ts), (indptr, nbr, eid, ats)):
        for g, w in zip(got, (adj.indptr, adj.nbr, adj.eid, adj.ts)):
            assert np.array_equal(g.cpu().numpy()[:len(w)], w)


def test_adjacency_refuses_an_id_outside_the_table():
    from orca_b200 import _lib
    from orca_b200.neighbor_finder import NeighborFinder
    src, dst, eidx, ts = _stream(70000, 100, True, 1)
    dst[66000] = 100
    with pytest.raises(_lib.OrcaError) as e:
        NeighborFinder.build_on_device(src, dst, eidx, ts, 100)
    assert e.value.code == 5


@pytest.mark.parametrize("q,k", [(1, 1), (3, 7), (257, 16), (1000, 17), (4097, 32)])
def test_neighbor_tables_from_host_arrays(q, k):
    from oracle import tgn_oracle
    from orca_b200.neighbor_finder import NeighborFinder
    src, dst, eidx, ts = _stream(5000, 300, True, 9)
    nf = NeighborFinder.build_on_device(src, dst, eidx, ts, 300)
    rs = np.random.RandomState(q)
    nodes, times = rs.randint(0, 300, q), rs.rand(q) * 2000 - 100
    got = nf.get_temporal_neighbor(nodes, times, k)
    want = [t.cpu().numpy() for t in nf.sample_device(nodes, times, k)[:3]]
    oracle = tgn_oracle.Adjacency(src, dst, eidx, ts, 300)
    for g, w in zip(got, want):
        assert g.dtype == w.dtype and np.array_equal(g, w)
    for i in range(0, q, 50):      # the last k entries before the query time, right-aligned
        lo, hi = oracle.indptr[nodes[i]], oracle.indptr[nodes[i] + 1]
        row = oracle.nbr[lo:hi][oracle.ts[lo:hi] < times[i]][-k:]
        assert np.array_equal(got[0][i], np.r_[np.zeros(k - len(row), np.int32), row])


def test_tables_that_callers_keep_hold_a_bounded_amount_of_page_locked_memory():
    """Tables of many calls, or one table of each, stay with the caller: page-locked up to a limit, ordinary arrays
    beyond it, with the same contents; what is dropped can be page-locked again."""
    from orca_b200.neighbor_finder import NeighborFinder
    src, dst, eidx, ts = _stream(5000, 300, True, 9)
    nf = NeighborFinder.build_on_device(src, dst, eidx, ts, 300)
    rs = np.random.RandomState(3)
    nodes, times = rs.randint(0, 300, 60000), rs.rand(60000) * 2000
    locked = lambda a: torch.from_numpy(a).is_pinned()
    want = [t.cpu().numpy() for t in nf.sample_device(nodes, times, 20)[:3]]
    for keep in (slice(0, 3), slice(1, 2)):      # all three tables, or the middle one, which holds its neighbours
        held, n = [], 0
        for _ in range(24):                      # 14.4 MB a call
            tables = nf.get_temporal_neighbor(nodes, times, 20)
            n += locked(tables[0])
            held += tables[keep]
            for t, w in zip(tables, want):
                assert np.array_equal(t, w)
        assert 2 <= n and n * 3 * 4 * nodes.size * 20 <= 256 << 20
        del tables
        held.clear()
        assert all(locked(t) for t in nf.get_temporal_neighbor(nodes, times, 20))
    with pytest.raises(Exception):
        nf.get_temporal_neighbor(nodes, times, 33)      # (a call that fails holds nothing)
    assert all(locked(t) for t in nf.get_temporal_neighbor(nodes, times, 20))


def test_neighbor_tables_for_every_form_of_query():
    """One node, a matrix of nodes, lists, strided and read-only arrays, ids and times of other types, more times than
    nodes: what a list of nodes with a time each gives.  A node without a time is an error."""
    from orca_b200.neighbor_finder import NeighborFinder
    src, dst, eidx, ts = _stream(5000, 300, True, 9)
    nf = NeighborFinder.build_on_device(src, dst, eidx, ts, 300)
    rs = np.random.RandomState(5)
    nodes, times = rs.randint(0, 300, 24), np.floor(rs.rand(24) * 1500)
    want = nf.get_temporal_neighbor(nodes, times, 7)
    frozen = nodes.copy()
    frozen.flags.writeable = False
    for n, t in ((nodes.reshape(4, 6), times.reshape(4, 6)), (list(nodes), list(times)), (frozen, times),
                 (np.repeat(nodes, 2)[::2], np.repeat(times, 3)[::3]), (nodes.astype(np.float32), times.astype(np.int64)),
                 (nodes, np.r_[times, 5.0]), (nodes.reshape(24, 1), times), (torch.from_numpy(nodes).cuda(), times),
                 (torch.from_numpy(np.repeat(nodes, 2)).int().cuda()[::2], torch.from_numpy(np.repeat(times, 2)).cuda()[::2]),
                 (np.asfortranarray(nodes.reshape(4, 6).astype(np.int32)), times.reshape(4, 6))):
        for g, w in zip(nf.get_temporal_neighbor(n, t, np.int64(7)), want):
            assert g.dtype == w.dtype and np.array_equal(g, w)
    for g, w in zip(nf.get_temporal_neighbor(int(nodes[3]), float(times[3]), 7), want):
        assert np.array_equal(g, w[3:4])
    for n, t in ((nodes, times[:-1]), (nodes.reshape(4, 6), times[0])):
        with pytest.raises(ValueError):
            nf.get_temporal_neighbor(n, t, 7)
    with pytest.raises(TypeError):
        nf.get_temporal_neighbor(nodes, times, 7.5)
