"""Tree launches whose CTAs take their items from a counter.  The counter has to be zero again after
each launch: the same engine searches new data several times (launched, captured, replayed), with
fewer items than CTAs, as many, one more, and several rounds.  Column sums and tops are the oracle's
bit for bit.  (Adds and maxima of float32 in the tree's own order: no tolerance.)"""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

# (rows, tiles of 1056 channels); 148 SMs hold 296 CTAs of 16 rows
CASES = [(2, 1), (4, 296), (8, 297), (16, 295), (16, 296), (16, 593)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"T{c[0]}_tiles{c[1]}")
def test_counter_is_left_at_zero(port_oracle, case):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    T, tiles = case
    N, foff, tsamp, md = tiles * 1056 - 3, -2.7939677e-6, 18.253611, 0.3
    dd = Dedopplerer(T, N, foff, tsamp)
    xt = torch.empty((T, N), dtype=torch.float32, device="cuda")
    for i in range(4):
        x = np.random.default_rng(100 * T + i).exponential(1.0, (T, N)).astype(np.float32)
        xt.copy_(torch.from_numpy(x))
        _, _, arrays = port_oracle.search(x, foff, tsamp, md, 0.0, 8.0, arrays=True)
        dd.search_batch_raw([xt], [-1], [0], md, 0.0, 8.0)
        np.testing.assert_array_equal(dd.channel_array("colsum").cpu().numpy(), arrays["colsum"])
        np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
    dd.close()


def test_last_round_in_quarters(port_oracle):
    """A dozen rounds and more: the last round's drift blocks run in smaller chunks."""
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    T, N, n, foff, tsamp, md = 16, 280 * 1056 + 5, 13, -2.7939677e-6, 18.253611, 4.0
    dd = Dedopplerer(T, N, foff, tsamp)
    x = np.random.default_rng(5).exponential(1.0, (T, N)).astype(np.float32)
    _, _, arrays = port_oracle.search(x, foff, tsamp, md, 0.0, 5.0, arrays=True)
    xt = torch.from_numpy(x).cuda()
    key = lambda hits: [(h.index, h.drift_steps, h.power) for h in hits]
    alone = key(dd.search_batch_raw([xt], [-1], [0], md, 0.0, 5.0)[0])
    np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
    assert alone
    for hits in dd.search_batch_raw([xt] * n, [-1] * n, list(range(n)), md, 0.0, 5.0):
        assert key(hits) == alone
    np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
    dd.close()
