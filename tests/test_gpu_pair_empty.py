"""A child without rows in the PAIR stage: with min_samples_leaf and min_child_weight 0 and a
negative min_split_gain a leaf may send all its rows to one side.  The empty child is weak (it
has no axis split) but has no rows to search; its with-pairs split must still be written, or the
next select reads what an earlier fit left in that memory.  Against the oracle; every sum of the
first tree is exact in FP64, so its ties are the reference's."""
import numpy as np
import pytest
from test_gpu_pair import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaves,extra", [(64, 8, {}), (4096, 31, {}), (512, 12, dict(wave_expand=0))])
def test_empty_child_takes_no_pair_split(native, oracle, n, leaves, extra):
    i = np.arange(n)
    X = np.stack([i % 2, (i // 2) % 2], 1).astype(np.float64)
    y = 2.0 * X[:, 0] + X[:, 1] - 1.5  # four cells, mean 0
    ts = i // 16
    # what the pool hands out next holds pair splits
    rng = np.random.default_rng(3)
    Z = rng.standard_normal((2000, 6))
    warm = native.Booster(n_estimators=2, max_leaves=leaves, horizon=1, pair_splits=1, goss=0)
    warm.fit(Z, np.sign(Z[:, 0] * Z[:, 1]), timestamps=np.arange(2000) // 50)
    params = dict(n_estimators=1, learning_rate=0.5, max_depth=8, max_leaves=leaves, horizon=1, objective="mse", goss=0,
                  random_state=1, pair_splits=1, min_samples_leaf=0, min_child_weight=0.0, min_split_gain=-1.0)
    b = native.Booster(**dict(params, **extra))
    b.fit(X, y, timestamps=ts)
    ref, h = oracle.oracle_fit(params, X, y, ts)
    codes, nb = oracle.oracle_codes(X, params)
    try:
        assert (ref.trees[0].n_samples == 0).any()
        _compare(b.trees(), ref.trees, codes, nb)
    finally:
        oracle.oracle_free(h)
