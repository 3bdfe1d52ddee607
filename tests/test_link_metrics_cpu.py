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


class _Streams:
    """A model whose streams are TGN's as far as the evaluation can see: hands the negatives of two batches on and then
    fails, or scores all of them."""

    def __init__(self, fails):
        from orca_b200.tgn import TGN
        self.fails, self.taken = fails, 0
        self.eval = lambda: self
        self.eval_epoch, self.eval_epoch_metrics = (f.__get__(self) for f in (TGN.eval_epoch, TGN.eval_epoch_metrics))

    def _eval_stream(self, sources, destinations, negatives, timestamps, edge_idxs, k, bs, *rest):
        for lo in range(0, len(sources), bs):
            if self.fails and lo == 2 * bs:
                raise RuntimeError("in the middle")
            self.taken += len(negatives[lo:lo + bs])
        return np.linspace(0.6, 0.9, len(sources), dtype=np.float32), np.full(len(sources), 0.5, np.float32)


def _evaluate(model, sampler, n=50, bs=10):
    import types
    from orca_b200.evaluation import eval_edge_prediction
    a = np.arange(n)
    data = types.SimpleNamespace(sources=a, destinations=a, timestamps=a, edge_idxs=a, n_interactions=n)
    return eval_edge_prediction(model, sampler, data, 10, bs)


@pytest.mark.parametrize("replace", ["sample_destinations", "random_state", "dst_list"])
def test_draws_that_can_fail_are_made_before_anything_is_scored(replace):
    """A RandEdgeSampler of which something was replaced is somebody else's: its third draw fails, and no batch has been
    handed to the model by then."""
    from orca_b200.evaluation import RandEdgeSampler

    class Third:
        calls = 0

        def count(self):
            self.calls += 1
            if self.calls == 3:
                raise KeyError("third draw")

        def randint(self, lo, hi, size):
            if hi == 100:
                self.count()
            return np.zeros(size, np.int64)

        def __len__(self):
            return 100

        def __getitem__(self, at):
            self.count()
            return at

    sampler, third = RandEdgeSampler(np.arange(5), np.arange(100), seed=3), Third()
    if replace == "sample_destinations":
        sampler.sample_destinations = lambda size: third[np.arange(size)]
    elif replace == "random_state":
        sampler.reset_random_state = lambda: setattr(sampler, "random_state", third)
    else:
        sampler.dst_list = third
    model = _Streams(fails=False)
    with pytest.raises(KeyError):
        _evaluate(model, sampler)
    assert model.taken == 0


@pytest.mark.parametrize("fails", [False, True])
def test_the_sampler_is_left_behind_all_draws_of_the_stream(fails):
    from orca_b200.evaluation import RandEdgeSampler
    want, sampler = (RandEdgeSampler(np.arange(5), np.arange(100), seed=3) for _ in range(2))
    for _ in range(5):
        want.sample(10)
    model = _Streams(fails)
    if fails:
        with pytest.raises(RuntimeError, match="in the middle"):
            _evaluate(model, sampler)
        assert model.taken == 20
    else:
        _evaluate(model, sampler)
        assert model.taken == 50
    assert np.array_equal(want.sample(20)[1], sampler.sample(20)[1])


def _model_taking(taken):
    from orca_b200.tgn import TGN

    class Model(TGN):
        def __init__(self):
            pass

        n_layers = 2

        def eval(self):
            return self

        def _eval_stream(self, sources, destinations, negatives, *rest):
            taken.append((type(negatives), np.array(negatives[:])))
            e = len(sources)
            return np.full(e, .75, np.float32), np.full(e, .25, np.float32)

    return Model()


@pytest.mark.parametrize("n,bs,plan,reuse,beside", [(740, 37, True, True, False), (25000, 1000, True, True, False),
                                                    (25001, 1000, True, True, True), (330, 10, True, True, True),
                                                    (740, 37, False, True, True), (740, 37, True, False, True)])
def test_negatives_of_one_group_are_drawn_before_it(n, bs, plan, reuse, beside):
    """Negatives are drawn beside the GPU's work only where there is some: the ids are the same either way."""
    import types
    from orca_b200.evaluation import RandEdgeSampler, _Drawn, eval_edge_prediction
    a, taken = np.arange(n), []
    data = types.SimpleNamespace(sources=a, destinations=a, timestamps=a, edge_idxs=a, n_interactions=n)
    eval_edge_prediction(_model_taking(taken), RandEdgeSampler(np.arange(5), np.arange(100), seed=3), data, 10, bs, reuse=reuse,
                         cache_plan=[a[:1]] * (-(-n // bs)) if plan else None)
    want = RandEdgeSampler(np.arange(5), np.arange(100), seed=3)
    (kind, ids), = taken
    assert (kind is _Drawn) == beside
    assert np.array_equal(ids, np.concatenate([want.sample(min(bs, n - i))[1] for i in range(0, n, bs)]))
