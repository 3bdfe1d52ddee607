"""Metrics of a scored stream (orca_link_metrics) against scikit-learn's, batch by batch, at sizes on both sides of
the sort's switch, with short last batches, ties and more than one thread."""
import numpy as np
import pytest
from sklearn.metrics import accuracy_score, average_precision_score, roc_auc_score

from orca_b200 import _lib, build


@pytest.mark.parametrize("n,bs,levels", [(1, 200, 0), (7, 1, 0), (127, 127, 0), (128, 128, 5), (401, 129, 3), (6000, 2000, 0),
                                         (5003, 1000, 40), (300000, 4096, 0), (50, 20, 1)])
def test_metrics_equal_sklearn(n, bs, levels):
    build.build()
    rs = np.random.RandomState(n)
    pos, neg = (rs.rand(n).astype(np.float32) ** p for p in (0.8, 1.2))
    if levels:
        pos, neg = (np.floor(a * levels) / levels for a in (pos, neg))
        pos, neg = pos.astype(np.float32), neg.astype(np.float32)
    nb = -(-n // bs)
    got = np.empty((nb, 3))
    assert _lib.lib().orca_link_metrics(pos.ctypes.data, neg.ctypes.data, n, bs, got.ctypes.data) == 0
    for i in range(nb):
        p, q = pos[i * bs:(i + 1) * bs], neg[i * bs:(i + 1) * bs]
        y, s = np.r_[np.ones(len(p)), np.zeros(len(p))], np.r_[p, q]
        want = (average_precision_score(y, s), roc_auc_score(y, s),
                accuracy_score(np.zeros(len(p)), np.argmax(np.stack([p, q], axis=1), axis=1)))
        np.testing.assert_allclose(got[i], want, rtol=1e-12)


def test_scores_that_are_not_finite_are_refused():
    build.build()
    for bad in (np.nan, np.inf):
        pos, neg, out = np.full(10, 0.5, np.float32), np.full(10, 0.5, np.float32), np.empty((1, 3))
        neg[3] = bad
        rc = _lib.lib().orca_link_metrics(pos.ctypes.data, neg.ctypes.data, 10, 10, out.ctypes.data)
        assert rc == _lib.E_BADARG


@pytest.mark.parametrize("n,bs", [(1, 5), (7, 7), (20, 6), (23, 1)])
def test_negatives_drawn_when_asked_for_are_those_drawn_at_once(n, bs):
    from orca_b200.evaluation import RandEdgeSampler, _Drawn
    at_once, lazily = (RandEdgeSampler(np.arange(5), np.arange(100), seed=3) for _ in range(2))
    want = np.concatenate([at_once.sample(min(bs, n - lo))[1] for lo in range(0, n, bs)])
    drawn = _Drawn(n, bs, lazily.sample_destinations)
    assert drawn.drawn == min(bs, n) and len(drawn) == n
    for lo in range(0, n, 3):
        assert np.array_equal(drawn[lo:lo + 3], want[lo:lo + 3]) and drawn.drawn < lo + 3 + bs
    assert np.array_equal(drawn[:], want)
    assert at_once.random_state.randint(1 << 30) == lazily.random_state.randint(1 << 30)
