"""How a tree launch cuts its drift blocks into chunks: searches too small for one round of CTAs, and
the last, partly filled round of larger ones, run chunks of fewer drift blocks.  The top path sums
and column sums are the oracle's bit for bit at any cut.  (Adds and maxima of float32 in the
tree's own order: no tolerance.)"""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

# (rows, channels): one tile, a tile and its neighbours, a few tiles with a ragged last one, and
# enough tiles that the last round alone is cut (16 rows: 296 CTAs of 1056 channels; 32: 148)
SHAPES = [(2, 1056), (4, 1057), (8, 5 * 1056 - 1), (16, 1055), (16, 3 * 1056 + 1), (16, 320 * 1056 + 37), (32, 2 * 1056),
          (32, 170 * 1056 + 5)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"T{s[0]}_N{s[1]}")
def test_cut_launches_match_oracle(port_oracle, shape):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    from seticore_b200.synthetic import SearchSpec, make_filterbank_numpy
    T, N = shape
    md = 4.0 if N < 10000 else 1.0
    spec = SearchSpec(T, N, tsamp=18.253611 * 16 / max(T, 16), max_drift=md, seed=900 + T, n_tones=2, tone_drift=1.0,
                      snr_threshold=8.0)
    x = make_filterbank_numpy(spec)
    _, _, arrays = port_oracle.search(x, spec.foff_mhz, spec.tsamp, md, 0.0, 8.0, arrays=True)
    dd = Dedopplerer(T, N, spec.foff_mhz, spec.tsamp)
    xt = torch.from_numpy(x).cuda()
    for n in (1, 3):  # alone, and several whose last tiles share the last round
        dd.search_batch_raw([xt] * n, [-1] * n, list(range(n)), md, 0.0, 8.0)
        np.testing.assert_array_equal(dd.channel_array("colsum").cpu().numpy(), arrays["colsum"])
        np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
    dd.close()
