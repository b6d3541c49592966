"""Rows that start anywhere: every phase of base address and row stride against 16 bytes gives the
oracle's sums bit for bit (adds and maxima of float32 in the tree's order: no tolerance), for
bands whose ends fall inside a 16-byte chunk and for fewer channels than a chunk, and the 16-bit
forms the same hits."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu

# (rows, channels, row stride - channels, first element)
SHAPES = [(4, 67, 0, 0), (8, 1057, 2, 1), (16, 1058, 1, 2), (16, 4099, 5, 3), (32, 2113, 3, 1), (64, 1501, 0, 3), (64, 2998, 1, 2),
          (128, 1203, 2, 1)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"T{s[0]}_N{s[1]}_pad{s[2]}_at{s[3]}")
def test_row_phases_match_oracle(port_oracle, shape):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200 import Dedopplerer
    from seticore_b200.synthetic import SearchSpec, make_filterbank_numpy
    T, N, pad, at = shape
    spec = SearchSpec(T, N, tsamp=18.253611 * 16 / max(T, 16), max_drift=2.0, seed=1300 + T + N, n_tones=2, tone_drift=1.0,
                      snr_threshold=6.0)
    x = make_filterbank_numpy(spec)
    _, _, arrays = port_oracle.search(x, spec.foff_mhz, spec.tsamp, 2.0, 0.0, 6.0, arrays=True)
    flat = torch.full((at + T * (N + pad) + 8,), float("nan"), device="cuda")  # nothing outside a row is read
    view = flat[at:at + T * (N + pad)].view(T, N + pad)[:, :N]
    view.copy_(torch.from_numpy(x))
    dd = Dedopplerer(T, N, spec.foff_mhz, spec.tsamp)
    want = [(h.index, h.drift_steps, h.power) for h in dd.search_raw(view, -1, 0, 2.0, 0.0, 6.0)]
    np.testing.assert_array_equal(dd.channel_array("top").cpu().numpy(), arrays["top"])
    np.testing.assert_array_equal(dd.channel_array("colsum").cpu().numpy(), arrays["colsum"])
    for precision in ("bf16", "fp16"):
        dd.set_precision(precision)
        assert [(h.index, h.drift_steps, h.power) for h in dd.search_raw(view, -1, 0, 2.0, 0.0, 6.0)] == want
    dd.close()
