"""Hit windows and drift recovery at the sizes where their kernels change form: windows of one warp
and of one block (512 channels either side of the line), windows wider than the band, and paths
of fewer than, exactly and more than sixteen rows.  Hits equal the oracle's: the same channels,
drifts and powers (bit for bit: the path sums keep the tree's order)."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

# (rows, channels, window size in channels)
SHAPES = [(8, 9000, 512), (8, 9000, 514), (16, 9001, 510), (16, 9001, 512), (16, 9001, 540), (16, 700, 1500), (32, 6000, 62),
          (32, 6000, 620), (64, 5000, 130), (64, 5003, 2200)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"T{s[0]}_N{s[1]}_w{s[2]}")
def test_windows_match_oracle(port_oracle, shape):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    from seticore_b200.synthetic import SearchSpec, make_filterbank_numpy
    T, N, w = shape
    spec = SearchSpec(T, N, tsamp=18.253611 * 16 / max(T, 16), seed=1100 + T + w, n_tones=12, tone_drift=0.2,
                      tone_snr=(8.0, 60.0), snr_threshold=4.0)
    # the drift limit whose window size is w: w = 2 * ceil(limit / resolution)
    res = abs(1e6 * spec.foff_mhz / ((T - 1) * spec.tsamp))
    spec.max_drift = (w // 2 - 0.5) * res
    x = make_filterbank_numpy(spec)
    want, wstats, _ = port_oracle.search(x, spec.foff_mhz, spec.tsamp, spec.max_drift, 0.0, 4.0, arrays=True)
    assert wstats["window_size"] == w and len(want) >= 1
    dd = Dedopplerer(T, N, spec.foff_mhz, spec.tsamp)
    got = dd.search_raw(torch.from_numpy(x).cuda(), -1, 0, spec.max_drift, 0.0, 4.0)
    dd.close()
    thr = float(wstats["threshold"])
    # the statistics' emulated variance may move a threshold tie to the other side
    tie = lambda p: abs(float(p) - thr) <= 1e-4 * abs(thr)  # noqa: E731
    g = {h.index: (h.drift_steps, np.float32(h.power)) for h in got if not tie(h.power)}
    r = {h["index"]: (h["drift_steps"], np.float32(h["power"])) for h in want if not tie(h["power"])}
    assert g == r
