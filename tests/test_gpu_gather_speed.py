"""Slices around hits are gathered at the speed of their size: narrow slices as fast as wide ones of as many
values, and large lists by the faster of the two ways to the host."""
import statistics
import time

import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu


def _seconds(x, rows, width, n):
    import torch
    from seticore_b200.dedoppler import gather_hit_slices
    bounds = [(k * 997, k * 997 + width) for k in range(n)]
    t = []
    for _ in range(40):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        gather_hit_slices(x, rows, x.shape[1], bounds)
        t.append(time.perf_counter() - t0)
    return statistics.median(t[10:])


def test_narrow_slices():
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    x = torch.rand((256, 1 << 20), device="cuda")
    # Measured 1.0; a warp per row of one value, 1.5.
    assert _seconds(x, 256, 1, 400) < 1.25 * _seconds(x, 1, 256, 400)


def test_large_lists_take_the_faster_way(monkeypatch):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import dedoppler
    x = torch.rand((2, 1 << 20), device="cuda")
    now = _seconds(x, 2, 5000, 100)  # 10^6 values
    monkeypatch.setattr(dedoppler, "_GATHER_PINNED_FLOATS", 0)
    # Through device memory; straight into host memory measured 1.6 times that.
    assert now < 1.25 * _seconds(x, 2, 5000, 100)
