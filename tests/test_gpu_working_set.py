"""The serving loop's admission figure (tgb_working_set_bytes) against what a call takes from the
device's memory pool: never less, and not much more than a fixed allowance on top of it, so that
requests neither run out of memory nor wait for memory that nobody uses."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

USED, USED_HIGH = 7, 8  # cudaMemPoolAttrUsedMemCurrent, cudaMemPoolAttrUsedMemHigh


def _pool():
    torch.cuda.init()
    torch.cuda.synchronize()
    rt = C.CDLL("libcudart.so.12")
    pool = C.c_void_p()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    return rt, pool


def _taken(call):
    """Bytes of the pool that the call held at once, beyond what was held before it."""
    rt, pool = _pool()
    v = C.c_uint64(0)
    assert rt.cudaMemPoolSetAttribute(pool, USED_HIGH, C.byref(v)) == 0
    before, high = C.c_uint64(), C.c_uint64()
    assert rt.cudaMemPoolGetAttribute(pool, USED, C.byref(before)) == 0
    call()
    assert rt.cudaMemPoolGetAttribute(pool, USED_HIGH, C.byref(high)) == 0
    return high.value - before.value


def _charged(native, b, kind, X):
    return native.lib().tgb_working_set_bytes(b._h, kind, X.shape[0], X.shape[1], 0 if X.dtype == np.float32 else 1)


@pytest.mark.parametrize("n,nf,f64,params", [
    (300, 3, False, {}), (60000, 40, True, dict(pair_splits=True)), (60000, 40, False, dict(pair_splits=True, max_leaves=200, wave_expand=0)),
    (250000, 64, False, dict(objective="pairwise")), (300000, 20, False, dict(hist_bits=8, max_leaves=255)),
    (300000, 100, False, dict(goss=0)), (200000, 16, True, dict(grow=0)), (30000, 300, False, dict(n_estimators=300))])
def test_a_call_stays_within_its_working_set(native, n, nf, f64, params):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, nf)).astype(np.float64 if f64 else np.float32)
    y = X[:, 0] + rng.standard_normal(n)
    b = native.Booster(**dict(dict(n_estimators=3, horizon=1, pair_splits=False), **params))
    fit = _taken(lambda: b.fit(X, y, timestamps=np.arange(n) // 100))
    slack = 64 << 20
    assert fit <= _charged(native, b, 0, X) <= 1.6 * fit + 2 * slack
    predict = _taken(lambda: b.raw_predict(X))
    assert predict <= _charged(native, b, 1, X) <= 2 * predict + 2 * slack
