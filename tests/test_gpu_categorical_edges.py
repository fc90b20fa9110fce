"""A fit's edges and vocabularies with categorical columns (numeric edges from the device binner, next to
the host's vocabularies) equal the host binner's, bit for bit: float32 and float64, sampled and whole
columns, infinities and signed zeros in either kind of column."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("bin_sample", [0, 3000, 262144])
def test_fit_edges_equal_host_binner(native, dtype, bin_sample):
    rng = np.random.default_rng(1)
    n, nf = 20000, 7
    X = rng.standard_normal((n, nf))
    X[:, 1] = rng.integers(0, 20, n)
    X[:, 2] = rng.choice([0.0, -0.0, 2.0, np.inf], n)
    X[:, 4] = rng.choice([0.0, -0.0, 5.0], n)
    X[rng.random(n) < 0.01, 5] = np.inf
    X[rng.random((n, nf)) < 0.02] = np.nan
    X = np.ascontiguousarray(X.astype(dtype))
    is_cat = np.array([0, 1, 1, 0, 0, 0, 1], np.int32)
    b = native.Booster(n_estimators=1, horizon=1, max_depth=2, bin_sample=bin_sample, random_state=7, goss=0)
    b.fit(X, np.nan_to_num(X[:, 0]).astype(np.float64), timestamps=np.arange(n) // 50, is_cat=is_cat)
    e, ne = np.zeros(nf * 256), np.zeros(nf, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    nb = native.lib().tgb_binner_fit_cat(p(X), 0 if dtype == np.float32 else 1, n, nf, p(is_cat), 255, 5, bin_sample, 7,
                                         p(e), p(ne))
    assert nb == b.info()["n_bins"]
    for f in range(nf):
        assert np.array_equal(b.edges(f).view(np.int64), e[256 * f: 256 * f + ne[f]].view(np.int64)), f
