"""Vocabularies of categorical features where the counting table hands over to the sorted column:
both signs of zero (std::sort's order decides which is kept), about 8,192 distinct values, infinities,
an empty column.  tgb_binner_fit_cat against the oracle's Binner::fit, bit for bit."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.parametrize("distinct", [1, 300, 8191, 8192, 8193, 12000])
@pytest.mark.parametrize("min_count", [1, 3])
def test_vocabulary_matches_oracle(native, oracle, distinct, min_count):
    rng = np.random.default_rng(distinct)
    n, nf, max_bin = 30000, 4, 255
    X = np.zeros((n, nf))
    X[:, 0] = np.arange(n) % distinct
    X[:, 1] = rng.choice([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf], n)
    X[:, 2] = np.nan
    X[:, 3] = rng.standard_normal(distinct)[rng.integers(0, distinct, n)]
    is_cat = np.ones(nf, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    e1, n1, e2, n2 = np.zeros(nf * 256), np.zeros(nf, np.int32), np.zeros(nf * 256), np.zeros(nf, np.int32)
    nb1 = native.lib().tgb_binner_fit_cat(p(X), 1, n, nf, p(is_cat), max_bin, min_count, 5000, 7, p(e1), p(n1))
    L = oracle.oracle_lib()
    L.orc_binner_fit_cat.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_int, C.c_int, C.c_int, C.c_uint32,
                                     C.c_void_p, C.c_void_p, C.c_void_p]
    nb2 = L.orc_binner_fit_cat(p(X), n, nf, p(is_cat), max_bin, min_count, 5000, 7, p(e2), p(n2), None)
    assert nb1 == nb2 and np.array_equal(n1, n2)
    assert np.array_equal(e1.view(np.int64), e2.view(np.int64))
