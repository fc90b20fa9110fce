"""The waves estimate a feature's gains and evaluate those that can win; the one-split loop evaluates
all.  Where the estimate must step aside: two neighbouring bins whose gains differ by about 2^-34
of themselves under a negative min_split_gain of 2^15 to 2^22 of them, where both round to one
number and the lower bin wins; and targets whose squares reach the ends of a double's range.  Both
loops on the same exact sums, equal bit for bit."""
import numpy as np
import pytest

from test_gpu_wave_edges import _same

pytestmark = pytest.mark.gpu


def _both(native, X, y, **params):
    trees = []
    for grow in (0, 1):
        b = native.Booster(**dict(dict(n_estimators=1, learning_rate=0.1, max_depth=2, max_leaves=2, horizon=1, random_state=1,
                                       min_samples_leaf=1, min_child_weight=0.0, l2=1.0, pair_splits=False, goss=0,
                                       iid_mode=True, grow=grow), **params))
        b.fit(X, y)
        trees.append(b.trees())
    _same(trees[0], trees[1])
    return trees[1]


@pytest.mark.parametrize("m", [64, 300])
def test_gains_that_gamma_makes_equal(native, m):
    # bin 1: m rows of -1, bin 2: one row of almost nothing, bin 3: m rows of 1.  A split before or
    # behind the middle row has the same hessians, and gains apart by twice its share of m.
    X = np.concatenate([np.zeros(m), [1.0], np.full(m, 2.0)])[:, None].astype(np.float32)
    taken = set()
    for share in np.arange(-37.0, -31.9, 0.5):
        y = np.concatenate([np.full(m, -1.0), [-m * 2.0**share], np.ones(m)])
        for k in np.arange(15.0, 22.1, 0.5):
            tree = _both(native, X, y, min_split_gain=-2.0 * m * 2.0**k)[0]
            assert tree.is_leaf.size == 3
            taken.add(int(tree.threshold[0]))
    assert len(taken) == 2  # the better bin, and the lower one where gamma makes the two equal


@pytest.mark.parametrize("scale", [1e-165, 1e-161, 1e-158, 1e-155, 1e-140, 1e130, 1e140, 1e152, 1e154, 1e156])
@pytest.mark.parametrize("l2", [1.0, 1e-25, 1e25])
def test_targets_at_the_ends_of_the_range(native, scale, l2):
    rng = np.random.default_rng(2)
    n = 400
    X = rng.integers(0, 30, (n, 3)).astype(np.float32)
    y = scale * (X[:, 0] + rng.standard_normal(n))
    _both(native, X, y, max_leaves=6, max_depth=4, l2=l2)
    _both(native, X, y, max_leaves=6, max_depth=4, l2=l2, min_split_gain=-scale * scale)
