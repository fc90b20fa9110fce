"""GOSS where the 32-bit sort keys tie: runs of tied keys with unlike |g| around the length that the
fix-up still orders itself (64).  Longer ones are reported and the fit is repeated with the 64-bit
sort; of a run of 65 the last row took itself for one of a short run and left a place of the order
without a row.  Against the oracle: all |g| of the first tree differ, so the samples are the same."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("run", [2, 63, 64, 65, 66, 127, 128, 129, 130])
def test_runs_of_tied_keys(native, oracle, run):
    rng = np.random.default_rng(run)
    n = 1200
    X = rng.standard_normal((n, 4))
    y = rng.standard_normal(n) * 3 + np.sign(X[:, 0])
    rows = rng.permutation(n)
    y[rows[:run]] = 1.75 + 1e-12 * rng.permutation(run)  # one key, unlike patterns, largest last or first
    y[rows[run:2 * run]] = -2.5 - 1e-12 * np.arange(run)
    ts = np.arange(n) // 40
    params = dict(n_estimators=1, learning_rate=0.1, max_depth=5, max_leaves=12, horizon=1, objective="mse", goss=1,
                  random_state=4, pair_splits=0, min_samples_leaf=5, iid_mode=1, goss_top=0.3, goss_other=0.2)
    b = native.Booster(**params)
    b.fit(X, y, timestamps=ts)
    assert b.fit_stats()["goss_refits"] == (1 if run > 64 else 0)
    ref, h = oracle.oracle_fit(params, X, y, ts)
    oracle.oracle_free(h)
    for a, r in zip(b.trees(), ref.trees, strict=True):
        for f in ("is_leaf", "feature", "threshold", "left", "right", "n_samples"):
            assert np.array_equal(getattr(a, f), getattr(r, f)), f
        np.testing.assert_allclose(a.values, r.values, rtol=0, atol=1e-9)
