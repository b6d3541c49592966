"""Batches of searches whose channel count is not a multiple of four: every search's arrays start on a
16-byte boundary all the same, so each search of the batch finds what it finds alone (its hits
are equal, power and SNR bit for bit), in every storage form and with whole-number power, whose
statistics take the exact order."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("T,N", [(8, 2051), (16, 2049), (16, 4101), (30, 3002), (64, 2053)])
def test_odd_batches_equal_single_searches(T, N, precision):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    Tr = 1 << (T - 1).bit_length()
    g = torch.Generator(device="cuda")
    g.manual_seed(T * N)
    xs = []
    for k in range(5):
        x = torch.zeros((Tr, N), device="cuda")
        x[:T].exponential_(1.0, generator=g).mul_(20.0)
        x[:T, 400 + 37 * k] += 200.0
        if k % 2:
            x.round_()
        xs.append(x)
    dd = Dedopplerer(T, N, 2.7939677e-6, 18.253611 * 16 / max(T, 16))
    dd.set_precision(precision)
    key = lambda hits: [(h.index, h.drift_steps, h.power, h.snr) for h in hits]  # noqa: E731
    alone = [key(dd.search_raw(x, -1, 0, 1.0, 0.0, 8.0)) for x in xs]
    assert all(alone)
    for _ in range(2):
        batch = dd.search_batch_raw(xs, [-1] * 5, list(range(5)), 1.0, 0.0, 8.0)
        assert [key(h) for h in batch] == alone
    dd.close()
