"""The statistics of a large batch of small searches run side by side: clusters small enough that one round
of CTAs holds them.  Device times of a batch against a smaller one that fits a round whatever the cluster."""
import statistics

import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu


def _search_ms(n, whole):
    import torch
    from seticore_b200 import Dedopplerer
    T, N, foff = 8, 16384, 2.7939677
    g = torch.Generator("cuda").manual_seed(n)
    x = torch.empty((n, T, N), device="cuda").exponential_(generator=g)
    if whole:  # many equal column sums: the statistics take the reference's own order
        x = (x * 4).floor()
    dd = Dedopplerer(T, N, foff * 1e-6, 18.25)
    ms = []
    for _ in range(30):
        dd.search_batch_raw(list(x), [-1] * n, list(range(n)), 0.2, 0.0, 200.0)
        ms.append(dd.last_stats().search_ms)
    assert dd.last_stats().order_exact == int(whole)
    dd.close()
    return statistics.median(ms[10:])


def test_exact_statistics_of_a_large_batch():
    if not has_gpu():
        pytest.skip("no CUDA device")
    # 15 searches fill one round of clusters of eight.  64 take 1.2 times as long with clusters of two,
    # and 3.4 times with eight.
    assert _search_ms(64, True) < 2 * _search_ms(15, True)


def test_statistics_of_a_large_batch():
    if not has_gpu():
        pytest.skip("no CUDA device")
    # 33 searches fill one round of clusters of eight.  37 take as long with clusters of four, and 1.38
    # times as long with eight.
    assert _search_ms(37, False) < 1.2 * _search_ms(33, False)


@pytest.mark.parametrize("n,tied", [(33, 2), (33, 15), (33, 16), (40, 33), (64, 64), (64, 0), (20, 20)])
def test_tied_searches_of_a_large_batch(n, tied):
    """Few and many tied searches of a batch, by either launch: every search's hits, whose SNR holds the
    deviation, are those of the search alone, launched, captured and replayed."""
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    T, N, foff = 4, 70001, 2.7939677
    g = torch.Generator("cuda").manual_seed(n + tied)
    x = torch.empty((n, T, N), device="cuda").exponential_(generator=g)
    pick = [k for k in range(n) if (k * 7) % n < tied]
    assert len(pick) == tied
    x[pick] = (x[pick] * 4).floor()
    one, dd = (Dedopplerer(T, N, foff * 1e-6, 18.25) for _ in range(2))
    key = lambda hits: [(h.index, h.drift_steps, h.power, h.snr) for h in hits]
    want = []
    for k in range(n):
        want.append(key(one.search_raw(x[k], -1, 0, 0.4, 0.0, 3.0)))
        assert one.last_stats().order_exact == int(k in pick)
    assert all(want)
    for _ in range(4):
        assert [key(h) for h in dd.search_batch_raw(list(x), [-1] * n, list(range(n)), 0.4, 0.0, 3.0)] == want
    one.close()
    dd.close()
