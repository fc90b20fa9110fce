"""tgb_partition where the tiles of 2,048 rows and the grid end: none, one, an edge, more tiles
than the grid has blocks, back-to-back calls through one workspace (a call's scatter reads its
rows while its count runs), and codes at odd columns and strides."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,stride,feature,listed", [
    (1, 16, 15, 1.0), (2047, 17, 16, 1.0), (2048, 33, 0, 1.0), (2049, 128, 64, 0.5), (700_001, 48, 31, 0.3),
    (4_000_003, 16, 5, 0.9)])
def test_partition_is_stable_at_the_edges(native, n, stride, feature, listed):
    import torch

    L, g = native.lib(), torch.Generator(device="cuda").manual_seed(n)
    codes = torch.randint(0, 64, (n, stride), device="cuda", dtype=torch.uint8, generator=g)
    rows = torch.nonzero(torch.rand(n, device="cuda", generator=g) < listed).flatten().to(torch.int32)
    k = rows.numel()
    size = L.tgb_partition_workspace_bytes(k)
    work = torch.empty(size, device="cuda", dtype=torch.uint8)
    a, b = torch.empty_like(rows), torch.empty_like(rows)
    left = torch.zeros(2, device="cuda", dtype=torch.int32)
    s = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def split(src, dst, f, thr, miss, at):
        native.check(L.tgb_partition(C.c_void_p(codes.data_ptr()), stride, C.c_void_p(src.data_ptr()), k, f, thr, miss,
                                     C.c_void_p(dst.data_ptr()), C.c_void_p(left.data_ptr() + 4 * at),
                                     C.c_void_p(work.data_ptr()), size, s))

    # the second call splits the first one's output, with nothing between them
    split(rows, a, feature, 20, 1, 0)
    split(a, b, (feature + 1) % stride, 40, 0, 1)
    c, r = codes.cpu().numpy(), rows.cpu().numpy()

    def expect(r, f, thr, miss):
        v = c[r, f]
        m = np.where(v == 0, bool(miss), v <= thr)
        return np.concatenate([r[m], r[~m]]), int(m.sum())

    ea, la = expect(r, feature, 20, 1)
    eb, lb = expect(ea, (feature + 1) % stride, 40, 0)
    assert left.tolist() == [la, lb]
    assert np.array_equal(a.cpu().numpy(), ea) and np.array_equal(b.cpu().numpy(), eb)
