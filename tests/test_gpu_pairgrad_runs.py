"""Pairwise gradients of panels of many short runs, which share warps and CTAs, against the same runs
a few at a time, which take a CTA each: equal bit for bit.  Runs around the sizes where the work
changes hands (8, 29, 48 rows), without rows, of equal targets, with NaN targets, long ones among
short ones; and whole fits on such panels against the oracle."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

FEW = 1000  # runs of a call that take a CTA each


def _call(native, y, p, start, length, order, per_call):
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    q = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    yd, pd, od = d(y), d(p), None if order is None else d(order)
    g = torch.full((len(y),), 7.0, dtype=torch.float64, device="cuda")
    h = torch.full((len(y),), 7.0, dtype=torch.float64, device="cuda")
    for k in range(0, len(start), per_call):
        s, m = d(start[k:k + per_call]), d(length[k:k + per_call])
        rows = int(length[k:k + per_call].sum())
        native.check(native.lib().tgb_grad_pairwise(q(yd), q(pd), q(s), q(m), q(od), s.numel(), rows, q(g), q(h), None))
        torch.cuda.synchronize()
    return g.cpu().numpy(), h.cpu().numpy()


@pytest.mark.parametrize("runs,lengths,kind", [
    (1037, [20], "plain"), (1500, [0, 1, 2, 8, 9, 28, 29, 30], "ties"), (8191, [1, 2, 3, 7, 8, 9], "nan"),
    (8192, [1, 2, 3, 7, 8], "plain"), (9000, [0, 1, 2, 8, 9, 17], "nan"), (10001, [1, 3, 4], "ordered"),
    (8500, [2, 3, 2, 3, 2, 3, 2, 29, 30, 2, 3, 1, 1, 1, 1, 48], "ordered"), (3000, [5, 700, 6, 2] + [9] * 60, "plain")])
def test_short_runs_equal_a_cta_a_run(native, runs, lengths, kind):
    rng = np.random.default_rng([runs, len(lengths)])
    length = np.resize(np.array(lengths, np.int32), runs)
    n = int(length.sum())
    start = (np.cumsum(length) - length).astype(np.int32)
    y, p = rng.standard_normal(n), 3 * rng.standard_normal(n)
    if kind == "ties":
        y = np.round(y)
    y[start[5]:start[5] + length[5]] = 0.25  # a run of equal targets
    if kind == "nan":
        y[rng.random(n) < 0.03] = np.nan
    order = rng.permutation(n).astype(np.int32) if kind == "ordered" else None
    got = _call(native, y, p, start, length, order, runs)
    want = _call(native, y, p, start, length, order, FEW)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("dates,rows", [(1200, 5), (8300, 3)])
def test_fit_on_short_dates_matches_oracle(native, oracle, dates, rows):
    rng = np.random.default_rng(dates)
    n = dates * rows
    X = rng.standard_normal((n, 4))
    y = X[:, 0] - 0.5 * X[:, 1] + 0.3 * rng.standard_normal(n)
    ts = np.arange(n) // rows
    params = dict(n_estimators=2, learning_rate=0.1, max_depth=4, max_leaves=8, horizon=1, objective="pairwise", goss=0,
                  random_state=1, pair_splits=0)
    b = native.Booster(**params)
    b.fit(X, y, timestamps=ts)
    ref, h = oracle.oracle_fit(params, X, y, ts)
    oracle.oracle_free(h)
    for a, r in zip(b.trees(), ref.trees, strict=True):
        assert np.array_equal(a.feature, r.feature) and np.array_equal(a.threshold, r.threshold)
        np.testing.assert_allclose(a.values, r.values, rtol=0, atol=1e-9)
    np.testing.assert_allclose(b.evals_result()["train"], ref.evals_train, rtol=0, atol=1e-9)
