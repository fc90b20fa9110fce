"""The PAIR search where its chunks, its ranking and its hash can go wrong: one chunk and many
chunks a child, two features, repeated columns (ties in the ranking of the features, where
std::sort's own order decides the pairs), few bins, per-row hessians and GOSS, many children a
wave.  Against the oracle restatement, values within 1e-9 as everywhere."""
import numpy as np
import pytest
from test_gpu_pair import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nf,copies,extra", [
    (600, 2, 0, {}), (5000, 40, 3, {}), (30000, 33, 0, dict(objective="pairwise")), (20000, 70, 5, dict(goss=1)),
    (9000, 12, 2, dict(max_bin=8)), (40000, 9, 0, dict(max_leaves=64, wave_expand=0, max_pair_splits_per_tree=20)),
    (9000, 6, 0, dict(pair_top_k=2))])
def test_pair_search_matches_oracle(native, oracle, n, nf, copies, extra):
    rng = np.random.default_rng([n, nf])
    X = rng.standard_normal((n, nf))
    X[rng.random((n, nf)) < 0.04] = np.nan
    for k in range(copies):  # repeated columns tie in every ranking
        X[:, nf - 1 - k] = X[:, k]
    y = np.sign(np.nan_to_num(X[:, 0]) * np.nan_to_num(X[:, 1])) + 0.5 * rng.standard_normal(n)
    ts = np.arange(n) // 100
    params = dict(n_estimators=3, learning_rate=0.1, max_depth=6, max_leaves=20, horizon=1, random_state=1,
                  pair_splits=1, objective="mse", goss=0)
    params.update(extra)
    b = native.Booster(**params)
    b.fit(X, y, timestamps=ts)
    ref_params = {k: v for k, v in params.items() if k != "wave_expand"}
    ref, h = oracle.oracle_fit(ref_params, X, y, ts)
    codes, nb = oracle.oracle_codes(X, ref_params)
    try:
        _compare(b.trees(), ref.trees, codes, nb)
    finally:
        oracle.oracle_free(h)
