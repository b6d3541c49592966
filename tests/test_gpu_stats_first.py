"""Statistics formed before the tree (batches of one or two searches) and after it (larger ones).
Column sums and tops are the oracle's bit for bit either way, and the statistics of a search do not
depend on the route.  (The same kernels on the same column sums: no tolerance.)"""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

# (rows, channels): one tile and a few, ragged; rows that the level path takes; enough tiles that the
# levels of a batch form the column sums
SHAPES = [(2, 1057), (16, 4093), (16, 40000), (32, 33001), (64, 4001), (64, 110003), (256, 5000)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"T{s[0]}_N{s[1]}")
@pytest.mark.parametrize("integers", [False, True], ids=["floats", "integers"])
def test_statistics_before_and_after_the_tree(port_oracle, shape, integers):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    T, N = shape
    foff, tsamp, md = -2.7939677e-6, 18.253611 * 16 / T, 1.0
    x = np.random.default_rng(T + N).exponential(1.0, (T, N)).astype(np.float32)
    if integers:  # repeated column sums: the exact statistics
        x = np.floor(4 * x)
    _, _, arrays = port_oracle.search(x, foff, tsamp, md, 0.0, 8.0, arrays=True)
    dd = Dedopplerer(T, N, foff, tsamp)
    xt = torch.from_numpy(x).cuda()
    seen = []
    for n in (1, 2, 3, 1):
        dd.search_batch_raw([xt] * n, [-1] * n, list(range(n)), md, 0.0, 8.0)
        np.testing.assert_array_equal(dd.channel_array("colsum").cpu().numpy(), arrays["colsum"])
        np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
        q = dd.last_stats()
        seen.append((q.median, q.mean, q.std_dev, q.order_exact))
    assert seen == [seen[0]] * 4
    assert integers <= bool(seen[0][3])
    dd.close()
