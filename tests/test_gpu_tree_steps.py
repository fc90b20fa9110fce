"""Trees whose waves end anywhere in the tree graph's steps (its straight waves, the IF nodes after
them, the loop): one expansion a wave, so that a tree of L leaves takes L - 1 waves or a few more,
trees that end early although many leaves are allowed, and batches of both.  Against the
one-split loop, bit for bit."""
import numpy as np
import pytest

from test_gpu_wave_edges import _case, _same

pytestmark = pytest.mark.gpu


def _fit(native, n, nf, **params):
    X, y, ts = _case(n, nf)
    b = native.Booster(**dict(dict(n_estimators=3, learning_rate=0.1, max_depth=9, horizon=1, random_state=3,
                                   min_samples_leaf=2, pair_splits=False, goss=0), **params))
    b.fit(X, y, timestamps=ts)
    return b


@pytest.mark.parametrize("leaves", [2, 3, 4, 5, 8, 9, 10, 16, 17, 18, 19, 40])
def test_one_expansion_a_wave(native, leaves):
    a = _fit(native, 3001, 5, max_leaves=leaves, wave_expand=1)
    assert a.fit_stats()["graph_used"] == 1
    _same(a.trees(), _fit(native, 3001, 5, max_leaves=leaves, grow=0).trees())


@pytest.mark.parametrize("leaves", [31, 255])
@pytest.mark.parametrize("extra", [dict(min_split_gain=1e9), dict(min_split_gain=200.0), dict(min_split_gain=20.0),
                                   dict(max_depth=1), dict(max_depth=2), dict(min_samples_leaf=700),
                                   dict(min_samples_leaf=200, objective="pairwise")])
def test_trees_that_end_early(native, leaves, extra):
    _same(_fit(native, 3001, 5, max_leaves=leaves, **extra).trees(),
          _fit(native, 3001, 5, max_leaves=leaves, grow=0, **extra).trees())


def test_batch_of_short_and_long_trees(native):
    sets = [dict(max_leaves=255, min_split_gain=1e9), dict(max_leaves=255), dict(max_leaves=2), dict(max_leaves=31, max_depth=2)]
    data = [_case(2000 + 500 * k, 5, k) for k in range(len(sets))]
    base = dict(n_estimators=3, learning_rate=0.1, max_depth=9, horizon=1, random_state=3, min_samples_leaf=2,
                pair_splits=False, goss=0)
    bs = [native.Booster(**dict(base, **p)) for p in sets]
    native.Booster.fit_batch(bs, *[list(c) for c in zip(*data)])
    for b, p, (X, y, ts) in zip(bs, sets, data):
        own = native.Booster(**dict(base, grow=0, **p))
        own.fit(X, y, timestamps=ts)
        _same(b.trees(), own.trees())
