"""tgb_hist_build where its splits and tiles can go wrong: values around the 2^39 boundary of the
split and up to the largest a caller may pass, few and many of them in a warp, sub-chunk and warp
remainders, ragged feature groups, sums added to what the outputs hold.  Exact integers, against
Python integers through numpy."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nf", [(1, 1), (31, 5), (33, 17), (1023, 16), (2049, 32), (4097, 33), (70001, 40)])
@pytest.mark.parametrize("kind", ["small", "edge", "few", "largest"])
def test_hist_build_is_exact(native, n, nf, kind):
    rng = np.random.default_rng([n, nf])
    total = n + 500
    stride = (nf + 15) // 16 * 16
    codes = np.zeros((total, stride), np.uint8)
    codes[:, :nf] = rng.integers(0, 256, (total, nf))
    codes[:, 0] = 7  # every row in one bin
    rows = rng.permutation(total)[:n].astype(np.int32)
    top = 62 - 1 - int(np.ceil(np.log2(max(2, n))))
    if kind == "small":
        g = rng.integers(-2**36, 2**36, total)
    elif kind == "edge":
        g = rng.choice([-2**39 - 1, -2**39, -2**39 + 1, 2**39 - 1, 2**39, 2**39 + 1, 0, -1, 1], total)
    elif kind == "few":
        g = rng.integers(-2**30, 2**30, total)
        at = rng.random(total) < 0.08
        g[at] = rng.integers(-2**(top - 1), 2**(top - 1), int(at.sum()))
    else:
        g = rng.integers(-2**top, 2**top, total)
    g = (g >> 10 << 10) if top > 52 and kind in ("few", "largest") else g  # exact as float64
    h = np.abs(g[::-1]).copy()
    ref = [np.full((nf, 256), 3, np.int64), np.full((nf, 256), 5, np.int64), np.full((nf, 256), 2, np.int32)]
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    q = lambda t: C.c_void_p(t.data_ptr())
    off = 0 if kind != "small" else 3  # a code matrix may start at any byte
    cd = torch.zeros(off + codes.size, dtype=torch.uint8, device="cuda")[off:]
    cd.copy_(d(codes.reshape(-1)))
    rd, gd, hd = d(rows), d(g.astype(np.float64)), d(h.astype(np.float64))
    out = [d(r) for r in ref]
    native.check(native.lib().tgb_hist_build(q(cd), stride, nf, q(rd), n, q(gd), q(hd), 0, 0, q(out[0]), q(out[1]),
                                             q(out[2]), None))
    torch.cuda.synchronize()
    for f in range(nf):
        b = codes[rows, f]
        np.add.at(ref[0][f], b, g.astype(np.float64).astype(np.int64)[rows])
        np.add.at(ref[1][f], b, h.astype(np.float64).astype(np.int64)[rows])
        np.add.at(ref[2][f], b, 1)
    for o, r in zip(out, ref):
        assert np.array_equal(o.cpu().numpy(), r)
