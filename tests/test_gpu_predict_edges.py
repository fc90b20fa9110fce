"""Predictions at the sizes where the kernel's row tiles, its batches of trees and the chunked
copies can go wrong, against a numpy walk of the exported trees (same sums in the same order: equal
to the last bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _walk(b, X, is_cat=None):
    n, nf = X.shape
    codes = np.zeros((n, nf), np.int64)
    for f in range(nf):
        e, v = b.edges(f), X[:, f].astype(np.float64)
        if is_cat is not None and is_cat[f]:
            k = np.minimum(np.searchsorted(e, v), len(e) - 1)
            codes[:, f] = np.where(e[k] == v, k + 1, 0)
        else:
            codes[:, f] = np.where(np.isnan(v), 0, np.searchsorted(e, v, side="right") + 1)
    info = b.info()
    out = np.full(n, info["init_score"])
    for t in b.trees():
        k = np.zeros(n, np.int64)
        while not t.is_leaf[k].all():
            c = codes[np.arange(n), np.where(t.is_leaf[k] != 0, 0, t.feature[k])]
            c2 = codes[np.arange(n), np.maximum(t.feature2[k], 0)]
            ml = t.missing_left[k] != 0
            left = np.where(c == 0, ml, c <= t.threshold[k])
            z = ((c * 2654435761 + c2 * 40503) & 0xffffffff) % info["n_bins"]
            left = np.where(t.split_type[k] == 1, np.where((c == 0) | (c2 == 0), ml, z <= t.threshold[k]), left)
            bit = (t.cat_left[k, c >> 6] >> (c & 63).astype(np.uint64)) & np.uint64(1)
            left = np.where(t.split_type[k] == 2, bit != 0, left)
            k = np.where(t.is_leaf[k] != 0, k, np.where(left, t.left[k], t.right[k]))
        out = out + b.params["learning_rate"] * t.values[k]
    return out


def _model(native, nf, **extra):
    rng = np.random.default_rng(nf)
    n = 3000
    X = rng.standard_normal((n, nf))
    X[rng.random((n, nf)) < 0.03] = np.nan
    is_cat = None
    if extra.pop("cat", False):
        is_cat = np.zeros(nf, np.int32)
        is_cat[-1] = 1
        X[:, -1] = rng.integers(0, 9, n)
    y = np.sign(np.nan_to_num(X[:, 0]) * np.nan_to_num(X[:, 1 % nf])) + np.nan_to_num(X[:, -1]) + 0.2 * rng.standard_normal(n)
    p = dict(n_estimators=37, learning_rate=0.1, max_depth=7, horizon=1, random_state=1, pair_splits=False, goss=0,
             min_samples_leaf=5)
    p.update(extra)
    b = native.Booster(**p)
    b.fit(X, y, timestamps=np.arange(n) // 30, is_cat=is_cat)
    return b, is_cat


def _rows(n, nf, dtype, cat):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, nf)).astype(dtype)
    X[rng.random((n, nf)) < 0.03] = np.nan
    if cat is not None:
        X[:, -1] = rng.integers(0, 11, n)
    return X


@pytest.mark.parametrize("nf,extra", [
    (1, {}), (6, {}), (40, dict(max_leaves=200, max_depth=12)), (17, dict(pair_splits=1, cat=True)),
    (9, dict(pair_splits=1)), (6600, dict(n_estimators=3)), (300, dict(n_estimators=70, max_leaves=4))])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_predict_matches_tree_walk(native, nf, extra, dtype):
    b, is_cat = _model(native, nf, **dict(extra))
    for n in (1, 31, 33, 1000) if nf > 1000 else (1, 32, 1000, 18945, 75777, 131073):
        if n * nf > 12_000_000:
            continue
        X = _rows(n, nf, dtype, is_cat)
        assert np.array_equal(b.raw_predict(X), _walk(b, X, is_cat)), n


def test_predict_follows_a_second_fit(native):
    """The layout kept for predictions belongs to the last fit, whatever the dtypes in between."""
    rng = np.random.default_rng(0)
    b, _ = _model(native, 6)
    X32 = _rows(500, 6, np.float32, None)
    X64 = _rows(500, 6, np.float64, None)
    for scale in (1.0, 3.0, 1.0):
        Xf = rng.standard_normal((2000, 6)) * scale
        b.fit(Xf, Xf[:, 0] + 0.1 * rng.standard_normal(2000), timestamps=np.arange(2000) // 20)
        for X in (X32, X64, X32):
            assert np.array_equal(b.raw_predict(X), _walk(b, X))
