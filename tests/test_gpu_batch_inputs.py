"""Searches of one call with data of their own: a launch that split, reordered or re-chunked its groups and
read one search's rows or raised another's tops would change their hits.  Every search's hits are those
of the same search alone, whose arrays other tests compare with the oracle.  (The same float32 adds and
maxima: no tolerance.)"""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

FOFF = 2.7939677  # Hz


def _inputs(T, N, n, seed):
    import torch
    g = torch.Generator("cuda").manual_seed(seed)
    rows = 1 << (T - 1).bit_length()
    out = []
    for _ in range(n):
        x = torch.empty((rows, N), device="cuda").exponential_(generator=g)
        x[T:] = 0.0
        out.append(x)
    return out


def _key(hits):
    return [(h.index, h.drift_steps, h.power, h.snr) for h in hits]


# (rows, channels, drift limit in Hz/s, searches in the call): the last round cut into quarters after a
# dozen rounds and more, with a group split and with whole groups; a part-filled round; groups of 32 rows; sums
# formed by the levels on the side streams; two searches with their statistics beside the tree
BATCHES = [(16, 280 * 1056 + 5, 4.0, 13), (16, 60 * 1056, 4.0, 64), (16, 50001, 4.0, 7), (32, 100003, 2.0, 5),
           (64, 105000, 0.3, 5), (16, 65536, 4.0, 2), (8, 200001, 4.0, 3)]


@pytest.mark.parametrize("shape", BATCHES, ids=lambda s: f"T{s[0]}_N{s[1]}_md{s[2]}_n{s[3]}")
def test_batch_searches_keep_their_own_data(shape):
    if not has_gpu():
        pytest.skip("no CUDA device")
    from seticore_b200 import Dedopplerer
    T, N, md, n = shape
    xs = _inputs(T, N, n, seed=T * N + n)
    tsamp = 18.253611 * 16 / T
    one, dd = (Dedopplerer(T, N, FOFF * 1e-6, tsamp) for _ in range(2))
    want = [_key(one.search_raw(x, -1, 0, md, 0.0, 5.0)) for x in xs]
    assert all(want) and len({tuple(w) for w in want}) == n
    for order in (list(range(n)), list(range(n))[::-1]):
        got = dd.search_batch_raw([xs[k] for k in order], [-1] * n, order, md, 0.0, 5.0)
        for k, hits in zip(order, got):
            assert _key(hits) == want[k], k
        # the first search's arrays are kept
        one.search_raw(xs[order[0]], -1, 0, md, 0.0, 5.0)
        for name in ("top", "colsum"):
            np.testing.assert_array_equal(dd.channel_array(name).cpu().numpy(), one.channel_array(name).cpu().numpy())
    one.close()
    dd.close()


def test_pool_searches_of_uneven_drift_ranges():
    """More than a dozen rounds of items, longest drift ranges last: the launch sorts its groups while it
    cuts the last round."""
    if not has_gpu():
        pytest.skip("no CUDA device")
    from seticore_b200 import Dedopplerer, SearchPool, SearchRequest
    T, tsamp, reqs, want = 16, 18.253611, [], []
    for k in range(16):
        N, md = 250000 + 1057 * k, 0.4 + 0.25 * k
        x, = _inputs(T, N, 1, seed=900 + k)
        reqs.append(SearchRequest(x, T, FOFF * 1e-6, tsamp, md, 0.0, 5.0))
        one = Dedopplerer(T, N, FOFF * 1e-6, tsamp)
        want.append(_key(one.search_raw(x, -1, 0, md, 0.0, 5.0)))
        one.close()
    assert all(want)
    pool = SearchPool()
    for _ in range(3):  # launched and tuned, captured, replayed
        assert [_key(h) for h in pool.search_raw(reqs)] == want
