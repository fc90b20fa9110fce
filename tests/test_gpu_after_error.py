"""A call that runs out of device memory reports it and leaves nothing behind: the next call of the same
thread works (the error used to stay with the CUDA runtime and failed the next launch's check)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_a_fit_after_one_out_of_memory(native):
    rng = np.random.default_rng(0)
    X = rng.standard_normal((200, 3))
    y, ts = X[:, 0] + 0.1 * rng.standard_normal(200), np.arange(200) // 10
    params = dict(n_estimators=2, horizon=1, pair_splits=False, goss=0, min_samples_leaf=5)
    want = native.Booster(**params)
    want.fit(X, y, timestamps=ts)
    # the trees' nodes alone would be 1.3 TB: the first allocation of that size is refused
    with pytest.raises(native.TideError, match="out of memory"):
        native.Booster(**dict(params, n_estimators=20_000_000, max_leaves=256)).fit(X, y, timestamps=ts)
    got = native.Booster(**params)
    got.fit(X, y, timestamps=ts)
    assert np.array_equal(got.raw_predict(X), want.raw_predict(X))


def test_a_batch_after_one_whose_set_up_fails(native):
    rng = np.random.default_rng(1)
    data = []
    for n in (3000, 200, 5000, 700):
        X = rng.standard_normal((n, 6)).astype(np.float32)
        data.append((X, X[:, 0] + 0.1 * rng.standard_normal(n), np.arange(n) // 10))
    params = dict(n_estimators=3, horizon=1, pair_splits=False, goss=1, min_samples_leaf=5)
    bs = [native.Booster(**params) for _ in data]
    bs[1].set_config(max_leaves=1)
    with pytest.raises(native.TideError, match="max_leaves"):
        native.Booster.fit_batch(bs, *[list(c) for c in zip(*data)])
    bs[1].set_config(max_leaves=31)
    native.Booster.fit_batch(bs, *[list(c) for c in zip(*data)])
    for b, (X, y, ts) in zip(bs, data):
        own = native.Booster(**params)
        own.fit(X, y, timestamps=ts)
        assert np.array_equal(b.raw_predict(X), own.raw_predict(X))
