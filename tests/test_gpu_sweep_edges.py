"""What a tree starts and ends with, against the oracle at the sizes where its tiles end: the
sample's rows around tiles of 4,096 and ends within 16 rows, the sweep's tiles of 512 rows with
few, 33 to 64 and more split columns, and prediction steps of 1,024 rows that cross buckets."""
import numpy as np
import pytest

from test_gpu_fit import _compare

pytestmark = pytest.mark.gpu


def _fit_both(native, oracle, n, nf, params, iid):
    rng = np.random.default_rng([n, nf])
    X = rng.standard_normal((n, nf)).astype(np.float32)
    w = rng.standard_normal(nf)
    y = np.tanh(X) @ w + 0.1 * rng.standard_normal(n)
    ts, ent = (None, None) if iid else (np.arange(n) // 9, np.arange(n) % 9)
    gpu = native.Booster(**params)
    gpu.fit(X, y, timestamps=ts, entity=ent)
    ref, h = oracle.oracle_fit(params, X.astype(np.float64), y, *(() if iid else (ts, ent)))
    try:
        _compare(gpu, ref)
    finally:
        oracle.oracle_free(h)


def test_smallest_sample(native):
    """65 rows, the fewest that are sampled: nodes of a few rows have splits that tie exactly (one
    partition mirrored by another feature), which the oracle's own summation order decides, so the
    one-split loop, exact as the waves are, gives the trees here."""
    rng = np.random.default_rng(65)
    X, y = rng.standard_normal((65, 5)).astype(np.float32), rng.standard_normal(65)
    trees = []
    for grow in (0, 1):
        b = native.Booster(n_estimators=4, learning_rate=0.1, max_depth=5, max_leaves=12, iid_mode=1, objective="mse",
                           goss=1, random_state=3, pair_splits=False, min_samples_leaf=2, grow=grow)
        b.fit(X, y)
        trees.append(b.trees())
    for a, b in zip(*trees, strict=True):
        assert a.n_samples[0] == 20  # ceil(0.2 n) of the largest and ceil(0.1 n) of the others
        for f in ("feature", "threshold", "left", "right", "n_samples", "cover", "values"):
            assert np.array_equal(getattr(a, f), getattr(b, f)), f


@pytest.mark.parametrize("n", [4095, 4096, 4097, 8207, 12304])
def test_sample_rows_at_tile_edges(native, oracle, n):
    params = dict(n_estimators=4, learning_rate=0.1, max_depth=5, max_leaves=12, iid_mode=1, objective="mse", goss=1,
                  random_state=3, pair_splits=False, min_samples_leaf=2)
    _fit_both(native, oracle, n, 5, params, True)


@pytest.mark.parametrize("n,nf,leaves", [(513, 3, 8), (9001, 60, 120), (7001, 120, 250), (33333, 7, 31)])
def test_sweep_and_prediction_steps(native, oracle, n, nf, leaves):
    params = dict(n_estimators=4, learning_rate=0.1, max_depth=9, max_leaves=leaves, horizon=1, objective="mse", goss=0,
                  random_state=3, pair_splits=False, min_samples_leaf=5)
    _fit_both(native, oracle, n, nf, params, False)
