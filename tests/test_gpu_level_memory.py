"""Level buffers: an engine of more than 32 rows holds what its shape needs when it is created, and grows
once calls whose drift range can use more keep coming.  Tops and column sums are the oracle's bit for bit
before and after."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,N", [(64, 1024), (200, 4099), (512, 1024)])
def test_buffers_grow_with_the_drift_range(port_oracle, T, N):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    foff, tsamp = 1e6 / 262144, 0.268435456
    Tr = 64 if T == 64 else 256 if T == 200 else 512
    x = np.zeros((Tr, N), dtype=np.float32)
    x[:T] = np.random.default_rng(T).exponential(1.0, (T, N))
    x[:T, 300] += 2.0
    xt = torch.from_numpy(x).cuda()
    dd = Dedopplerer(T, N, foff * 1e-6, tsamp)
    row = (N + 1055) // 1056 * 1056 + 2048
    created = dd.memoryUsage()
    # four pairs, each buffer of two drift blocks' plane rows (one above 256 rows), and less than a
    # megabyte and a half of other scratch
    assert created < 4 * 8 * (2 if Tr <= 256 else 1) * Tr * row + (3 << 19)
    used = []
    for nmax in (0.5, 60.5, 0.5):  # 2, 122 and 2 drift blocks
        md = nmax * foff / tsamp
        _, _, want = port_oracle.search(x, foff * 1e-6, tsamp, md, 0.0, 5.0, arrays=True)
        for _ in range(19 if nmax > 1 else 3):  # launched, captured, replayed, and so again once the buffers grew
            dd.search_raw(xt, -1, 0, md, 0.0, 5.0)
            np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), want["top"])
            np.testing.assert_array_equal(dd.channel_array("colsum").cpu().numpy(), want["colsum"])
        used.append(dd.memoryUsage())
    grown = used[1] - used[0]
    assert grown == (used[2] - used[0])
    assert (grown > 0) == (T <= 256)  # more rows take one drift block at a time
    assert used[1] < 300 << 20
    dd.close()
