"""Bin codes at the shapes and edges where the lane mapping and the halving search can go wrong:
1 to 33 and 70 features (several rows a warp, a ragged last group), 0, 1, 254 and 255 edges,
repeated, infinite, NaN and unsorted edges, categorical columns; values that are NaN, infinite,
signed zeros and exactly on an edge.  Against numpy's searchsorted where the edges are sorted and a
restatement of libstdc++'s upper_bound / lower_bound otherwise."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _bound(e, v, upper):
    first, size = 0, len(e)
    while size > 0:
        half = size >> 1
        mid = first + half
        go = (not v < e[mid]) if upper else (e[mid] < v)
        if go:
            first, size = mid + 1, size - half - 1
        else:
            size = half
    return first


def _code(e, v):
    return 0 if v != v else (_bound(e, v, True) + 1) & 255


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nf", [1, 2, 3, 5, 16, 17, 31, 32, 33, 70])
def test_transform_matches_upper_bound(native, dtype, nf):
    rng = np.random.default_rng(nf)
    n = 1037 if nf > 3 else 3001
    X = np.round(rng.standard_normal((n, nf)) * 8).astype(dtype) / 8
    special = np.array([np.nan, np.inf, -np.inf, 0.0, -0.0], dtype)
    X[rng.random((n, nf)) < 0.1] = 0.0
    at = rng.random((n, nf)) < 0.1
    X[at] = special[rng.integers(0, 5, int(at.sum()))]
    E = np.full((nf, 256), -7.0, dtype)  # what follows a feature's edges is not read
    ne = np.zeros(nf, np.int32)
    for f in range(nf):
        ne[f] = [254, 0, 1, 255, 7, 128, 127, 64][f % 8]
        e = np.sort(np.round(rng.standard_normal(ne[f]) * 8) / 8)
        if f % 5 == 1 and ne[f] > 3:
            e[[0, -1]] = -np.inf, np.inf
        if f % 7 == 3 and ne[f] > 3:
            e[ne[f] // 2] = np.nan
        if f % 7 == 5 and ne[f] > 3:
            e = e[::-1]
        E[f, : ne[f]] = e
    stride = (nf + 15) // 16 * 16
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    p = lambda t: C.c_void_p(t.data_ptr())
    Xd, Ed, nd = d(X), d(E), d(ne)
    codes = torch.full((n, stride), 77, dtype=torch.uint8, device="cuda")
    native.check(native.lib().tgb_bin_transform(p(Xd), 0 if dtype == np.float32 else 1, n, nf, p(Ed), p(nd), p(codes),
                                                stride, None))
    torch.cuda.synchronize()
    got = codes.cpu().numpy()
    want = np.array([[_code(E[f, : ne[f]], X[i, f]) for f in range(nf)] for i in range(n)], np.uint8)
    assert np.array_equal(got[:, :nf], want)
    assert (got[:, nf:] == 0).all()
