"""sc_dd_gather_columns on ranges that hold nothing: an empty range, or one whose end lies before its begin,
writes nothing."""
import ctypes

import numpy as np
import pytest

from tests.conftest import has_gpu


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [3, 9])
def test_empty_and_reversed_ranges(rows):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200._capi import lib
    x = torch.rand((rows, 100), device="cuda")
    ranges = torch.tensor([7, 7, 50, 10, 20, 60, 60, 59], dtype=torch.int32, device="cuda")
    offsets = torch.tensor([0, 0, 1, 0], dtype=torch.int64, device="cuda")
    out = torch.full((rows * 40 + 2,), -1.0, device="cuda")
    assert lib().sc_dd_gather_columns(ctypes.c_void_p(x.data_ptr()), 100, rows, 100, ctypes.c_void_p(ranges.data_ptr()),
                                      ctypes.c_void_p(offsets.data_ptr()), 4, ctypes.c_void_p(out.data_ptr()), None) == 0
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    np.testing.assert_array_equal(got[1:-1].reshape(rows, 40), x[:, 20:60].cpu().numpy())
    assert got[0] == got[-1] == -1.0
