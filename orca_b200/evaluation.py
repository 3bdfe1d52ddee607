"""``eval_edge_prediction`` with the signature and return value of the reference's evaluation loop
(evaluation/evaluation.py:6-47): mean average precision, AUC and accuracy over the batches of the
stream, one uniform negative destination per positive edge drawn batch by batch from the sampler.

The reference calls the model once per batch and brings the scores back per batch; here the whole
stream goes through ``TGN.eval_epoch_metrics`` -- one call.  The sampler is consumed exactly as the
reference consumes it (same draws, same order): before the first batch, or, where it is this module's
own and nothing of it has been replaced, for a longer stream while the GPU works on the batches before.  The metrics are
those of scikit-learn, per batch as in the reference, computed by the library.
"""
from __future__ import annotations

import math

import numpy as np

from . import _lib
from .tgn import TGN


class RandEdgeSampler:
    """Uniform negative sampler with the interface of utils/util.py:68-87: sample(size) draws `size`
    source indices and then `size` destination indices from one seeded RandomState over the sorted
    unique id lists."""

    def __init__(self, src_list, dst_list, seed=None):
        self.seed = seed
        self.src_list = np.unique(src_list)
        self.dst_list = np.unique(dst_list)
        self.random_state = np.random.RandomState(seed) if seed is not None else np.random

    def sample(self, size):
        src_index = self.random_state.randint(0, len(self.src_list), size)
        dst_index = self.random_state.randint(0, len(self.dst_list), size)
        return self.src_list[src_index], self.dst_list[dst_index]

    def sample_destinations(self, size):
        """The destinations of sample(size): the sources are drawn all the same, so that the state moves on alike."""
        self.random_state.randint(0, len(self.src_list), size)
        return self.dst_list[self.random_state.randint(0, len(self.dst_list), size)]

    def reset_random_state(self):
        self.random_state = np.random.RandomState(self.seed)


class _Drawn:
    """The negatives of a stream, one draw a batch in the stream's order, made when a batch is first asked for (TGN.eval_epoch
    packs a group of batches while the GPU works on the one before)."""

    def __init__(self, n, batch_size, draw):
        self.ids, self.batch_size, self.draw, self.drawn = np.empty(n, dtype=np.int64), batch_size, draw, 0
        self[:1]      # (a sampler that cannot draw says so before anything is scored)

    def __len__(self):
        return len(self.ids)

    def __getitem__(self, part):
        ids, bs, draw, at, upto, end = self.ids, self.batch_size, self.draw, self.drawn, part.stop, len(self.ids)
        if upto is None or upto > end:
            upto = end
        while at < upto:
            to = min(end, at + bs)
            ids[at:to] = draw(to - at)
            self.drawn = at = to
        return ids[part]


def _plain(sampler):
    """Whether the sampler's draws are this module's own all through, on its own lists and generator: such a draw does not
    fail once the first one has succeeded, and nobody sees when it is made."""
    return type(sampler) is RandEdgeSampler and not {"sample", "sample_destinations"} & vars(sampler).keys() and \
        type(sampler.random_state) is np.random.RandomState and \
        all(type(ids) is np.ndarray and ids.dtype.kind in "iu" for ids in (sampler.src_list, sampler.dst_list))


def eval_edge_prediction(model, negative_edge_sampler, data, n_neighbors, batch_size, reuse=True, cache_plan=None):
    assert negative_edge_sampler.seed is not None
    negative_edge_sampler.reset_random_state()
    model = model.eval()
    # (only the destinations are used; this module's own sampler can draw the sources without looking them up)
    draw = negative_edge_sampler.sample_destinations if type(negative_edge_sampler) is RandEdgeSampler else \
        lambda size: negative_edge_sampler.sample(size)[1]
    n = data.n_interactions
    nb = math.ceil(n / batch_size)
    negatives = _Drawn(n, batch_size, draw)
    # A stream that goes through the model as one group (orca_group_sizes: at most 32 batches, 76 k rows on 148 SMs, three an edge)
    # has nothing to draw beside.  20 batches of 37 edges: 831 us, drawn beside it 850; 40 of 200, two groups: 1630, drawn beside it 1530.
    one_group = nb <= 32 and n <= 25000 and reuse and (cache_plan is not None or getattr(model, "n_layers", 2) == 1)
    own = not one_group and \
        all(getattr(getattr(model, f, None), "__func__", None) is getattr(TGN, f) for f in ("eval_epoch", "eval_epoch_metrics"))
    if not own or not _plain(negative_edge_sampler):
        negatives = negatives[:]      # (somebody else's: all draws before the first batch, as the reference's caller sees it)
    try:
        # per batch, as the reference does; the positive "wins" when its score is not below the negative's
        # (evaluation/evaluation.py:39-40)
        stream = (data.sources[:n], data.destinations[:n], negatives, data.timestamps[:n], data.edge_idxs[:n], n_neighbors,
                  batch_size, cache_plan)
        if getattr(model.eval_epoch, "__func__", None) is TGN.eval_epoch:
            m = model.eval_epoch_metrics(*stream, reuse=reuse)
        else:       # (a model with an eval_epoch of its own: its scores count)
            pos, neg = model.eval_epoch(*stream, reuse=reuse)
            m = np.empty((nb, 3))
            rc = _lib.lib().orca_link_metrics(pos.ctypes.data, neg.ctypes.data, n, batch_size, m.ctypes.data)
            if rc == _lib.E_BADARG:
                raise ValueError(_lib.lib().orca_last_error().decode())
            _lib.check(rc)
    finally:
        negatives[:]      # (the sampler is left behind all draws of the stream, also where that fails half-way)
    val_ap, val_auc, val_acc = np.mean(m, axis=0)
    return val_ap, val_auc, val_acc
