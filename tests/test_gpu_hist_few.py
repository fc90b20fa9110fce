"""tgb_hist_build around the size where a few rows go straight to the output (1,024 rows, 2^18
(row, feature) pairs): exact on both sides, as in test_gpu_hist_edges.py."""
import pytest

from test_gpu_hist_edges import test_hist_build_is_exact as _exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nf", [(2, 1), (1024, 3), (1025, 3), (1024, 256), (1024, 257), (87, 3000), (88, 3000)])
@pytest.mark.parametrize("kind", ["small", "few", "largest"])
def test_hist_build_is_exact_around_the_few(native, n, nf, kind):
    _exact(native, n, nf, kind)
