"""Pairwise gradients at the run lengths where the residue classes change shape (one class up to 48
rows, classes of 24 to 36 above, classes that take the shared room of several warps), with tied
targets, saturated differences and NaN targets, in row order and through an order.  Against the
statements of objective.cpp:179-219 in numpy, within 1e-12 of the sum of the magnitudes (the
exponential differs by an ulp)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 24, 25, 29, 30, 36, 37, 41, 47, 48, 49, 50, 71, 72, 95, 96, 119, 120, 143, 144, 800, 1777]


def _reference(y, p):
    m = len(y)
    step = max(1, m // 24) if m > 48 else 1
    g, h, mag = np.zeros(m), np.full(m, 1e-6), np.full(m, 1e-6)
    for a in range(m):
        for b in range(a % step, m, step):
            if b == a or y[a] == y[b]:
                continue
            hi = y[a] > y[b]
            s = (p[a] - p[b]) if hi else (p[b] - p[a])
            e = np.exp(min(max(s, -30.0), 30.0))
            dy = abs(y[a] - y[b])
            dyw = 1e-6 if not dy > 1e-6 else dy
            lam, d2 = -1.0 / (1.0 + e) * dyw, e / ((1 + e) * (1 + e)) * dyw
            g[a] += lam if hi else -lam
            h[a] += d2
            mag[a] += abs(lam) + d2
    return g, h, mag


@pytest.mark.parametrize("kind", ["plain", "ties", "nan", "ordered"])
def test_pairwise_gradients(native, kind):
    rng = np.random.default_rng(5)
    n = sum(LENGTHS)
    y = rng.standard_normal(n)
    p = rng.standard_normal(n) * 3
    if kind == "ties":
        y, p = np.round(y), p * 20
    if kind == "nan":
        y[rng.random(n) < 0.02] = np.nan
    start = (np.cumsum(LENGTHS) - LENGTHS).astype(np.int32)
    order = rng.permutation(n).astype(np.int32) if kind == "ordered" else None
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    q = lambda t: None if t is None else C.c_void_p(t.data_ptr())
    yd, pd, sd, ld = d(y), d(p), d(start), d(np.array(LENGTHS, np.int32))
    od = None if order is None else d(order)
    g, h = torch.zeros(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    native.check(native.lib().tgb_grad_pairwise(q(yd), q(pd), q(sd), q(ld), q(od), len(LENGTHS), n, q(g), q(h), None))
    torch.cuda.synchronize()
    g, h = g.cpu().numpy(), h.cpu().numpy()
    for s, m in zip(start, LENGTHS):
        rows = np.arange(s, s + m) if order is None else order[s:s + m]
        rg, rh, mag = _reference(y[rows], p[rows])
        assert np.all(np.abs(g[rows] - rg) <= 1e-12 * mag), m
        assert np.all(np.abs(h[rows] - rh) <= 1e-12 * mag), m
