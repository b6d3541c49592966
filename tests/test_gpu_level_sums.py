"""Column sums formed by the levels' first pass (many tiles: alone a dozen per SM, beside others two) and
by their own launch (fewer), and the levels' passes that hold drift block 0 first, last or alone.
Column sums and top path sums are the oracle's bit for bit."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

# (rows, channels, drift limit in Hz/s at 2.79 Hz and 18.25 * 16 / T s per row, searches in one call)
SHAPES = [(64, 105000, 0.3, 2), (64, 105000, 0.3, 1), (64, 626001, 0.3, 1), (128, 104193, 1.5, 3), (64, 104192, 4.0, 2)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"T{s[0]}_N{s[1]}_md{s[2]}_n{s[3]}")
def test_level_sums_match_oracle(port_oracle, shape):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    T, N, md, n = shape
    foff, tsamp = 2.7939677e-6, 18.253611 * 16 / T
    rng = np.random.default_rng(T + N)
    x = rng.standard_exponential((T, N), dtype=np.float32) * np.float32(1e9)
    _, _, arrays = port_oracle.search(x, foff, tsamp, md, 0.0, 20.0, arrays=True)
    dd = Dedopplerer(T, N, foff, tsamp)
    xt = torch.from_numpy(x).cuda()
    for _ in range(2):
        # the first search of the call is the one whose arrays are kept
        dd.search_batch_raw([xt] * n, [-1] * n, list(range(n)), md, 0.0, 20.0)
        np.testing.assert_array_equal(dd.channel_array("colsum").cpu().numpy(), arrays["colsum"])
        np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
    dd.close()
