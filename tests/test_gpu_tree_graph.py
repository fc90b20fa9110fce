"""A tree as one graph launch against the same kernels enqueued by the host: fits alone and
batched (branches of the graph), every objective, the draws of several trees (odd and even
position buffers), stochastic rounding by tree, and one tree only.  Equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("is_leaf", "feature", "threshold", "left", "right", "missing_left", "n_samples", "depth", "value", "gain",
          "values", "cover", "prefix")


def _data(n, nf, seed):
    rng = np.random.default_rng([seed, n, nf])
    X = rng.standard_normal((n, nf)).astype(np.float32)
    y = X[:, 0] * X[:, -1] + 0.5 * rng.standard_normal(n)
    return X, y, np.arange(n) // 11, np.arange(n) % 11


def _same(a, b):
    assert np.array_equal(a.evals_result()["train"], b.evals_result()["train"])
    for p, q in zip(a.trees(), b.trees(), strict=True):
        for f in FIELDS:
            assert np.array_equal(getattr(p, f), getattr(q, f), equal_nan=getattr(p, f).dtype.kind == "f"), f


@pytest.mark.parametrize("params", [
    dict(), dict(goss=1), dict(goss=1, hist_bits=8), dict(goss=1, hist_bits=16, objective="pairwise"),
    dict(objective="pairwise", goss=1, n_estimators=1), dict(goss=1, pair_splits=True), dict(max_leaves=200)],
    ids=["mse", "goss", "goss8", "pairwise16", "pairwise_one_tree", "pair", "leaves200"])
@pytest.mark.parametrize("sizes", [(5003,), (700, 20011, 5003)], ids=["one", "three"])
def test_tree_graph_equals_host_launches(native, params, sizes):
    p = dict(n_estimators=5, learning_rate=0.1, max_depth=8, horizon=1, objective="mse", goss=0, pair_splits=False,
             random_state=5)
    p.update(params)
    got = []
    for graph in (1, 0):
        data = [_data(n, 19, k) for k, n in enumerate(sizes)]
        bs = [native.Booster(graph=graph, **p) for _ in sizes]
        if len(sizes) == 1:
            X, y, ts, ent = data[0]
            bs[0].fit(X, y, timestamps=ts, entity=ent)
        else:
            native.Booster.fit_batch(bs, *[list(c) for c in zip(*data)])
        assert bs[0].fit_stats()["graph_used"] == graph
        got.append(bs)
    for a, b in zip(*got):
        _same(a, b)
