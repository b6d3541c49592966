"""The statistics' clusters at the sizes where their CTA count changes (4, 8 or 16 CTAs by channel count
and batch size) and the exact statistics' pieces of 4096 terms at their edges, against the oracle:
median and mean exact, the deviation within the emulation's 1e-4 for distinct values and bit for bit
for repeated ones (whole numbers), as for every other size."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

SIZES = [64, 4095, 4096, 4097, 8192, 8193, 16384, 16385, 20481, 40961]


def _stats(dd, torch, xs):
    if len(xs) == 1:
        dd.search_raw(torch.from_numpy(xs[0]).cuda(), -1, 0, 1.0, 0.0, 10.0)
    else:
        dd.search_batch_raw([torch.from_numpy(x).cuda() for x in xs], [-1] * len(xs), list(range(len(xs))), 1.0, 0.0, 10.0)
    return dd.last_stats()


@pytest.mark.parametrize("whole", [False, True], ids=["distinct", "whole"])
@pytest.mark.parametrize("n", SIZES)
def test_cluster_sizes_match_oracle(port_oracle, n, whole):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    rng = np.random.default_rng(n + whole)
    xs = []
    for k in range(12):  # alone, and a batch large enough for clusters of eight
        x = np.zeros((2, n), np.float32)
        x[0] = rng.integers(0, 9 + k, n) if whole else rng.exponential(1.0, n) * 1e9
        xs.append(x)
    dd = Dedopplerer(2, n, 2.7939677e-6, 18.253611)
    for batch in (xs[:1], xs):
        g = _stats(dd, torch, batch)
        _, w = port_oracle.search(xs[0], 2.7939677e-6, 18.253611, 1.0, 0.0, 10.0)
        assert np.float32(g.median) == np.float32(w["median"])
        assert np.float32(g.mean).view(np.uint32) == np.float32(w["mean"]).view(np.uint32)
        if g.order_exact:
            assert np.float32(g.std_dev).view(np.uint32) == np.float32(w["std_dev"]).view(np.uint32)
        else:
            assert not whole or n == 64
            assert abs(g.std_dev - w["std_dev"]) <= 1e-4 * abs(w["std_dev"])
    dd.close()
