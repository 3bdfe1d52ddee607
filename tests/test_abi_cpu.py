"""CPU-side checks of the C-ABI library: it loads, exports every function the header declares,
rejects bad arguments with an error code and message, and the host-side adjacency build matches
the oracle.  No GPU is needed (no kernel is launched)."""
import ctypes
import os
import re
import subprocess
import sys

import numpy as np
import pytest

from helpers import graph
from orca_b200 import _lib, build
from oracle import tgn_oracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def L():
    build.build()
    return _lib.lib()


def _declared():
    text = open(os.path.join(ROOT, "include", "orca_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(orca_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported_and_bound(L):
    names = _declared()
    assert len(names) >= 20
    for n in names:
        assert hasattr(L, n), f"{n} is declared in include/orca_b200.h but not exported"
        assert n in _lib.SYMBOLS, f"{n} has no ctypes signature in orca_b200/_lib.py"
    assert sorted(_lib.SYMBOLS) == names


def test_bad_arguments_return_codes(L):
    assert L.orca_version() >= 1
    rc = L.orca_sample_topk(None, None, None, None, 10, None, None, 4, None, 10, None, None, None, None, None, None)
    assert rc == 1
    assert b"orca_sample_topk" in L.orca_last_error()
    assert L.orca_eval_workspace_bytes(0, 0, 10, 100) == -1
    assert L.orca_eval_workspace_bytes(200, 600, 10, 1501) > 0


@pytest.mark.parametrize("spec", ["t_nb2", "t_bip2", "c1"])
def test_csr_build_host_matches_oracle(L, spec):
    g = graph(spec)
    E, n = g.n_edges, g.n_nodes
    indptr = np.empty(n + 1, dtype=np.int64)
    nbr = np.empty(2 * E, dtype=np.int32)
    eid = np.empty(2 * E, dtype=np.int32)
    ts = np.empty(2 * E, dtype=np.float64)
    src, dst, eidx = (np.ascontiguousarray(a, dtype=np.int64) for a in (g.sources, g.destinations, g.edge_idxs))
    rc = L.orca_csr_build_host(src.ctypes.data, dst.ctypes.data, eidx.ctypes.data, g.timestamps.ctypes.data, E, n,
                               indptr.ctypes.data, nbr.ctypes.data, eid.ctypes.data, ts.ctypes.data)
    assert rc == 0
    adj = tgn_oracle.Adjacency(g.sources, g.destinations, g.edge_idxs, g.timestamps, n)
    assert np.array_equal(indptr, adj.indptr)
    assert np.array_equal(nbr, adj.nbr) and np.array_equal(eid, adj.eid) and np.array_equal(ts, adj.ts)


def test_csr_build_host_unsorted_stream_and_ties(L):
    rs = np.random.RandomState(0)
    E, n = 5000, 60
    src = rs.randint(1, n, E).astype(np.int64)
    dst = rs.randint(1, n, E).astype(np.int64)
    ts = rs.randint(0, 50, E).astype(np.float64)   # unsorted, many equal times, self loops allowed
    eidx = np.arange(1, E + 1, dtype=np.int64)
    indptr = np.empty(n + 1, dtype=np.int64)
    nbr = np.empty(2 * E, dtype=np.int32)
    eid = np.empty(2 * E, dtype=np.int32)
    ats = np.empty(2 * E, dtype=np.float64)
    rc = L.orca_csr_build_host(src.ctypes.data, dst.ctypes.data, eidx.ctypes.data, ts.ctypes.data, E, n,
                               indptr.ctypes.data, nbr.ctypes.data, eid.ctypes.data, ats.ctypes.data)
    assert rc == 0
    adj = tgn_oracle.Adjacency(src, dst, eidx, ts, n)
    assert np.array_equal(indptr, adj.indptr)
    assert np.array_equal(nbr, adj.nbr) and np.array_equal(eid, adj.eid) and np.array_equal(ats, adj.ts)
    bad = src.copy()
    bad[3] = n + 5
    rc = L.orca_csr_build_host(bad.ctypes.data, dst.ctypes.data, eidx.ctypes.data, ts.ctypes.data, E, n,
                               indptr.ctypes.data, nbr.ctypes.data, eid.ctypes.data, ats.ctypes.data)
    assert rc == 5


def test_no_fallback_without_cuda():
    import torch
    if torch.cuda.is_available():
        pytest.skip("a GPU is present")
    from orca_b200.history import History
    with pytest.raises(RuntimeError):
        History(10, 172, device="cuda")
    with pytest.raises(RuntimeError):
        History(10, 172, device="cpu")


LIMITED = """
import ctypes, resource, sys
import numpy as np
from orca_b200 import _lib
L = _lib.lib()
n, nodes = 300000, 8 << 20
pos, neg, out = np.linspace(0.1, 0.9, n).astype(np.float32), np.full(n, 0.5, np.float32), np.empty((74, 3))
want = out.copy()
ids, ts = np.zeros(1, np.int64), np.zeros(1)
indptr, adj = np.zeros(nodes + 1, np.int64), [np.zeros(2, t) for t in (np.int32, np.int32, np.float64)]
args = [a.ctypes.data for a in (ids, ids, ids, ts)] + [1, nodes] + [a.ctypes.data for a in (indptr, *adj)]
for i in range(74):     # (one batch a call: no threads yet, whose stacks would be kept)
    m = min(4096, n - 4096 * i)
    assert L.orca_link_metrics(pos[4096 * i:].ctypes.data, neg[4096 * i:].ctypes.data, m, 4096, want[i:].ctypes.data) == 0
# room for small allocations, not for another thread's stack or for 64 MB
size = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
resource.setrlimit(resource.RLIMIT_AS, (size + (6 << 20),) * 2)
rc = {"metrics": lambda: L.orca_link_metrics(pos.ctypes.data, neg.ctypes.data, n, 4096, out.ctypes.data),
      "csr": lambda: L.orca_csr_build_host(*args), "plan": lambda: L.orca_plan_host(
          0, ids.ctypes.data, ids.ctypes.data, 1, 1, 1, adj[0].ctypes.data, nodes, 1, 0, adj[1].ctypes.data, 2,
          indptr.ctypes.data, out.ctypes.data)}[sys.argv[1]]()
print("rc", rc, bool((out == want).all()))
"""


@pytest.mark.parametrize("entry,said", [("metrics", "rc 0 True"), ("csr", "rc 4"), ("plan", "rc 4")])
def test_no_exception_leaves_an_entry_point(entry, said):
    """Threads that cannot be started and host memory that is not there end neither the process (the shares are done by
    the calling thread) nor go unsaid (an error code)."""
    build.build()
    env = dict(os.environ, OMP_NUM_THREADS="1", OPENBLAS_NUM_THREADS="1", MALLOC_ARENA_MAX="1")
    r = subprocess.run([sys.executable, "-c", LIMITED, entry], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and said in r.stdout, (r.returncode, r.stdout, r.stderr[-2000:])


@pytest.mark.parametrize("bs,nb,k", [(1, 1, 1), (37, 32, 5), (200, 20, 10), (2000, 11, 32)])
def test_one_layer_has_no_room_for_embeddings_that_nobody_reads(L, bs, nb, k):
    """A group of a one-layer model leaves its rows to the scores as pairs; with two layers (here the recursion that recomputes
    no neighbours) every row has its embedding (688 bytes) and an operand image of it (192 columns of four bytes) beside that."""
    one, two = (L.orca_group_workspace_bytes(bs, nb, k, 0, 0, 5000, layers, 1) for layers in (1, 2))
    assert two - one >= 3 * bs * nb * (688 + 768) - 2 * 256


def test_version_of_the_prepared_operands(L, monkeypatch):
    """Weights are packed for one layout: header, library and package name the same one, a library of another is refused."""
    text = open(os.path.join(ROOT, "include", "orca_b200.h")).read()
    assert int(re.search(r"#define ORCA_VERSION (\d+)", text).group(1)) == L.orca_version() == _lib.VERSION
    monkeypatch.setattr(_lib, "VERSION", _lib.VERSION + 1)
    monkeypatch.setattr(_lib, "_lib", None)
    with pytest.raises(ImportError, match="interface version"):
        _lib.lib()
