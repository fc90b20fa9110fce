"""Batched growth against the one-split loop at the sizes where a wave kernel's tiling can go
wrong: row counts at the edges of the partition's 2048-row tiles, one to a few hundred
rows, ragged feature groups, few and many leaves.  Both loops sum exact integers, so the trees
are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(n, nf, seed=0):
    rng = np.random.default_rng([seed, n, nf])
    X = rng.standard_normal((n, nf)).astype(np.float32)
    X[:, 0] = np.round(X[:, 0] * 2)
    X[rng.random((n, nf)) < 0.05] = np.nan
    y = np.nan_to_num(X[:, 0]) - np.nan_to_num(X[:, -1]) + 0.3 * rng.standard_normal(n)
    return X, y, np.arange(n) // 7


def _same(a, b):
    assert len(a) == len(b)
    for t, (p, q) in enumerate(zip(a, b)):
        for f in ("is_leaf", "feature", "threshold", "left", "right", "missing_left", "n_samples", "depth", "value",
                  "gain", "values", "cover", "prefix"):
            # l2 = 0 gives NaN values at nodes without rows (0 / 0) in both loops
            assert np.array_equal(getattr(p, f), getattr(q, f), equal_nan=getattr(p, f).dtype.kind == "f"), (t, f)


@pytest.mark.parametrize("n,nf,leaves,extra", [
    (65, 1, 4, {}), (2047, 3, 31, {}), (2048, 33, 31, {}), (2049, 16, 31, {}), (4097, 17, 255, {}),
    (30011, 40, 255, dict(wave_expand=0)), (12289, 70, 255, dict(wave_expand=0, objective="pairwise")),
    (6144, 65, 8, {}), (20481, 31, 31, dict(goss=1)), (4096, 32, 2, {}),
    (9001, 40, 31, dict(objective="pairwise")), (70001, 96, 31, dict(objective="pairwise", goss=1))])
def test_waves_equal_one_split_loop(native, n, nf, leaves, extra):
    X, y, ts = _case(n, nf)
    p = dict(n_estimators=4, learning_rate=0.1, max_depth=8, max_leaves=leaves, horizon=1, random_state=3,
             min_samples_leaf=2, pair_splits=False, goss=0)
    p.update(extra)
    trees = []
    for grow in (0, 1):
        b = native.Booster(**dict(p, grow=grow))
        b.fit(X, y, timestamps=ts)
        trees.append(b.trees())
    _same(trees[0], trees[1])


@pytest.mark.parametrize("extra", [
    {}, dict(l2=0.0, min_child_weight=0.0), dict(l2=1e-40, min_child_weight=0.0), dict(min_split_gain=1e-3),
    dict(min_split_gain=-1e30), dict(min_child_weight=40.0), dict(l2=1e32), dict(objective="pairwise", l2=0.0)])
@pytest.mark.parametrize("kind", ["ties", "wide", "constant"])
def test_split_choice_equals_one_split_loop(native, kind, extra):
    """The waves estimate a feature's gains before they evaluate the few that can win, the
    one-split loop evaluates all.  Ties inside and across features (few values, repeated
    columns, a symmetric target), targets of very different magnitudes, a constant target, and
    the parameters at which the estimate must not be trusted."""
    rng = np.random.default_rng(11)
    n = 6000
    X = rng.integers(-3, 4, (n, 6)).astype(np.float32)
    X[:, 4] = X[:, 1]
    X[:, 5] = rng.standard_normal(n)
    X[rng.random(n) < 0.1, 2] = np.nan
    y = {"ties": np.sign(X[:, 1]) * np.sign(np.nan_to_num(X[:, 2])), "wide": 1e12 * X[:, 0] + 1e-6 * X[:, 5],
         "constant": np.full(n, 0.25)}[kind].astype(np.float64)
    p = dict(n_estimators=3, learning_rate=0.1, max_depth=6, horizon=1, random_state=1, min_samples_leaf=1,
             pair_splits=False, goss=0)
    p.update(extra)
    trees = []
    for grow in (0, 1):
        b = native.Booster(**dict(p, grow=grow))
        b.fit(X, y, timestamps=np.arange(n) // 20)
        trees.append(b.trees())
    _same(trees[0], trees[1])
