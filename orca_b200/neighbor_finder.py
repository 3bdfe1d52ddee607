"""Temporal neighbour finder on the GPU, with the interface of the reference's jitclass
(utils/util.py:91-151): ``get_neighbor_finder(data)``, ``NeighborFinder.find_before`` and
``NeighborFinder.get_temporal_neighbor`` keep their names, argument meaning and return dtypes.

The per-node Python lists of the reference become one time-sorted CSR (indptr int64, neighbour
int32, edge id int32, timestamp float64) resident in HBM, built there by ``orca_csr_build``;
``find_before`` copies the slice it returns to the host.
"""
from __future__ import annotations

import collections
import operator
import threading

import numpy as np
import torch

from . import _lib


class _Lent:
    """Bytes of page-locked memory that returned tables and plans hold, over the process: at most `limit` of them."""

    def __init__(self, limit):
        self.limit, self.held = limit, 0
        self.back = collections.deque()     # (what came back; filled by __del__, which must not wait for a lock)
        self.lock = threading.Lock()

    def take(self, n):
        """A share of n bytes, which comes back when it and the arrays made from it are gone; None: there is no room."""
        with self.lock:
            while self.back:
                self.held -= self.back.popleft()
            if self.held + n > self.limit:
                return None
            self.held += n
        return _Share(self.back, n)


class _Share:
    __slots__ = ("back", "n", "pin", "__array_interface__")

    def __init__(self, back, n):
        self.back, self.n = back, n

    def array(self, pin):
        """The page-locked tensor of bytes as an array that keeps this share."""
        self.pin = pin
        self.__array_interface__ = {"data": (pin.data_ptr(), False), "shape": (pin.numel(),), "typestr": "|u1", "version": 3}
        return np.asarray(self)

    def __del__(self):
        self.back.append(self.n)


class NeighborFinder:
    PINNED_TABLE = 64 << 20     # bytes of one returned table up to which it stays in page-locked memory
    LENT = _Lent(256 << 20)     # and of all that callers hold: a few calls' tables of the largest size

    def __init__(self, node_to_neighbors, node_to_edge_idxs, node_to_edge_timestamps, device="cuda"):
        """Same arguments as utils/util.py:123-126: per-node arrays, each already sorted by time."""
        lens = np.fromiter((len(a) for a in node_to_neighbors), dtype=np.int64, count=len(node_to_neighbors))
        indptr = np.zeros(len(lens) + 1, dtype=np.int64)
        np.cumsum(lens, out=indptr[1:])
        cat = lambda lst, dt: (np.concatenate([np.asarray(a, dtype=dt) for a in lst]) if len(lst) and indptr[-1]
                               else np.zeros(0, dtype=dt))
        self._init_csr(indptr, cat(node_to_neighbors, np.int32), cat(node_to_edge_idxs, np.int32),
                       cat(node_to_edge_timestamps, np.float64), device)

    @classmethod
    def from_csr(cls, indptr, nbr, eid, ts, device="cuda"):
        self = cls.__new__(cls)
        self._init_csr(indptr, nbr, eid, ts, device)
        return self

    def _init_csr(self, indptr, nbr, eid, ts, device):
        self.device = _lib.require_cuda(device)
        self.n_nodes = len(indptr) - 1
        self.indptr = torch.from_numpy(np.ascontiguousarray(indptr, dtype=np.int64)).to(self.device)
        # one spare element keeps the pointers valid for an empty graph
        pad = lambda a, dt: np.ascontiguousarray(a, dtype=dt) if len(a) else np.zeros(1, dtype=dt)
        self.adj_nbr = torch.from_numpy(pad(nbr, np.int32)).to(self.device)
        self.adj_eid = torch.from_numpy(pad(eid, np.int32)).to(self.device)
        self.adj_ts = torch.from_numpy(pad(ts, np.float64)).to(self.device)

    @classmethod
    def build_on_device(cls, sources, destinations, edge_idxs, timestamps, n_nodes, device="cuda"):
        """The adjacency of an edge stream, sorted on the GPU (utils/util.py:91-105)."""
        self = cls.__new__(cls)
        self.device = dev = _lib.require_cuda(device)
        self.n_nodes = int(n_nodes)
        E = len(sources)
        src, dst, eidx = (np.ascontiguousarray(a, dtype=np.int64) for a in (sources, destinations, edge_idxs))
        ts = np.ascontiguousarray(timestamps, dtype=np.float64)
        if not len(src) == len(dst) == len(eidx) == len(ts):
            raise ValueError("sources, destinations, edge_idxs and timestamps must have one length")
        L = _lib.lib()
        with torch.cuda.device(dev):
            new = torch.empty if E else torch.zeros      # (one spare element keeps the pointers of an empty graph valid)
            self.indptr = torch.empty(self.n_nodes + 1, dtype=torch.int64, device=dev)
            self.adj_nbr = new(max(2 * E, 1), dtype=torch.int32, device=dev)
            self.adj_eid = new(max(2 * E, 1), dtype=torch.int32, device=dev)
            self.adj_ts = new(max(2 * E, 1), dtype=torch.float64, device=dev)
            ws = torch.empty(max(L.orca_csr_build_workspace_bytes(E, self.n_nodes), 256), dtype=torch.uint8, device=dev)
            pin = torch.empty(max(L.orca_csr_build_pinned_bytes(E), 1), dtype=torch.uint8, pin_memory=True)
            stream = torch.cuda.current_stream(dev)
            rc = L.orca_csr_build_from_host(src.ctypes.data, dst.ctypes.data, eidx.ctypes.data, ts.ctypes.data, E,
                                            self.n_nodes, pin.data_ptr(), pin.numel(), self.indptr.data_ptr(),
                                            self.adj_nbr.data_ptr(), self.adj_eid.data_ptr(), self.adj_ts.data_ptr(),
                                            ws.data_ptr(), ws.numel(), stream.cuda_stream)
            stream.synchronize()                         # (the pinned chunks go back to their pool)
            _lib.check(rc)
        return self

    # --- utils/util.py:129-131
    def find_before(self, src_idx, cut_time):
        L = _lib.lib()
        node = torch.tensor([int(src_idx)], dtype=torch.int32, device=self.device)
        t = torch.tensor([float(cut_time)], dtype=torch.float64, device=self.device)
        cnt = torch.empty(1, dtype=torch.int32, device=self.device)
        _lib.check(L.orca_find_before(self.indptr.data_ptr(), self.adj_ts.data_ptr(), self.n_nodes,
                                      node.data_ptr(), t.data_ptr(), 1, cnt.data_ptr(),
                                      _lib.stream_ptr(self.device)))
        i = int(cnt.item())
        b = int(self.indptr[int(src_idx)].item())
        return (self.adj_nbr[b:b + i].cpu().numpy(), self.adj_eid[b:b + i].cpu().numpy(),
                self.adj_ts[b:b + i].cpu().numpy())

    # --- utils/util.py:134-151
    def get_temporal_neighbor(self, source_nodes, timestamps, n_neighbors):
        """Returns (neighbors int32 [Q,K], edge_idxs int32 [Q,K], edge_times float32 [Q,K]) as NumPy
        arrays: the K most recent interactions strictly before each query time, right-aligned,
        zero-padded on the left."""
        k = operator.index(n_neighbors)
        host = not isinstance(source_nodes, torch.Tensor) and not isinstance(timestamps, torch.Tensor)
        if host:
            nodes, ts = np.asarray(source_nodes), np.asarray(timestamps)
            host = nodes.ndim == 1 and ts.shape == nodes.shape
        q = nodes.size if host else 0
        table = 4 * q * k
        # The tables are returned in the page-locked memory that they were copied to: a fresh pageable array of a few
        # MB costs more in page faults than the whole call (40 k queries of ten: 195 us so, 860 on the general path).
        # Tables too large for that, more of them than callers may hold, inputs that are already on the GPU, of other
        # shapes than one list of nodes with a time each, and empty queries take the general path.
        out = (12 * q + 15) // 16 * 16 + 16
        share = None
        if 0 < table <= self.PINNED_TABLE:
            share = self.LENT.take(1 << (out + 3 * table - 1).bit_length())      # (the pool's blocks are powers of two)
        if share is None:
            nbr, eid, et, _ = self.sample_device(source_nodes, timestamps, n_neighbors)
            return nbr.cpu().numpy(), eid.cpu().numpy(), et.cpu().numpy()
        nodes, ts = np.ascontiguousarray(nodes, dtype=np.int64), np.ascontiguousarray(ts, dtype=np.float64)
        pin = torch.empty(out + 3 * table, dtype=torch.uint8, pin_memory=True)
        dev = torch.empty(out + 3 * table, dtype=torch.uint8, device=self.device)
        with torch.cuda.device(self.device):
            _lib.check(_lib.lib().orca_sample_topk_host(
                self.indptr.data_ptr(), self.adj_nbr.data_ptr(), self.adj_eid.data_ptr(), self.adj_ts.data_ptr(),
                self.n_nodes, nodes.ctypes.data, ts.ctypes.data, q, k, pin.data_ptr(), dev.data_ptr(), dev.numel(),
                _lib.stream_ptr(self.device)))
        h = share.array(pin)
        part = lambda i, dt: h[out + i * table:out + (i + 1) * table].view(dt).reshape(q, k)
        return part(0, np.int32), part(1, np.int32), part(2, np.float32)

    def sample_device(self, source_nodes, timestamps, n_neighbors, want_delta=False):
        """Same as get_temporal_neighbor but the tables stay on the device (torch tensors);
        also returns the fused time differences when asked."""
        k = n_neighbors if n_neighbors > 0 else 1
        nodes = torch.as_tensor(np.asarray(source_nodes), dtype=torch.int32).to(self.device) \
            if not isinstance(source_nodes, torch.Tensor) else source_nodes.to(self.device, torch.int32)
        ts = torch.as_tensor(np.asarray(timestamps), dtype=torch.float64).to(self.device) \
            if not isinstance(timestamps, torch.Tensor) else timestamps.to(self.device, torch.float64)
        nodes, ts, q = nodes.contiguous(), ts.contiguous(), nodes.numel()
        if ts.numel() < q:
            raise ValueError("every source node needs a timestamp")
        nbr = torch.zeros((q, k), dtype=torch.int32, device=self.device)
        eid = torch.zeros((q, k), dtype=torch.int32, device=self.device)
        et = torch.zeros((q, k), dtype=torch.float32, device=self.device)
        dt = torch.zeros((q, k), dtype=torch.float32, device=self.device) if want_delta else None
        if q and n_neighbors > 0:
            status = torch.zeros(4, dtype=torch.int32, device=self.device)
            L = _lib.lib()
            _lib.check(L.orca_sample_topk(self.indptr.data_ptr(), self.adj_nbr.data_ptr(),
                                          self.adj_eid.data_ptr(), self.adj_ts.data_ptr(), self.n_nodes,
                                          nodes.data_ptr(), ts.data_ptr(), q, None, k, nbr.data_ptr(),
                                          eid.data_ptr(), et.data_ptr(), _lib.ptr(dt), status.data_ptr(),
                                          _lib.stream_ptr(self.device)))
            _lib.check(L.orca_read_status(None, status.data_ptr(), None, _lib.stream_ptr(self.device)))
        return nbr, eid, et, dt


def get_neighbor_finder(data, max_node_idx=None, device="cuda"):
    """utils/util.py:91-105: every interaction is listed under both endpoints, each node's list
    stably sorted by time.  `data` needs .sources, .destinations, .edge_idxs, .timestamps."""
    src, dst = np.asarray(data.sources), np.asarray(data.destinations)
    if max_node_idx is None:
        max_node_idx = int(max(src.max(), dst.max())) if len(src) else 0
    return NeighborFinder.build_on_device(src, dst, data.edge_idxs, data.timestamps, int(max_node_idx) + 1,
                                          device=device)
