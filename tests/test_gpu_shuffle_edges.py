"""The device's draws of a shuffle where many words are rejected: ranges of tens to hundreds of
millions of values (one to some twenty rejections in a block of 624 words), and ends of a range
within a block.  The host sampler, itself held against std::shuffle, gives the prefix."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,keep,seed", [
    (65536, 65536, 1), (65536 + 623, 1000, 2), (65536 + 624, 1000, 3), (65536 + 625, 1, 4), (9_999_991, 200_000, 5),
    (40_000_003, 5000, 6), (150_000_001, 3000, 7), (300_000_007, 2000, 8)])
def test_device_draws_equal_host_draws(native, m, keep, seed):
    import torch

    out = torch.empty(keep, dtype=torch.int32, device="cuda")
    native.check(native.lib().tgb_shuffled_prefix_device(m, keep, seed, C.c_void_p(out.data_ptr()), None))
    torch.cuda.synchronize()
    ref = np.zeros(keep, np.int32)
    native.check(native.lib().tgb_shuffled_prefix(m, keep, seed, ref.ctypes.data_as(C.c_void_p)))
    assert np.array_equal(out.cpu().numpy(), ref)
