"""Slices around hits (gather_hit_slices) at the edges of its forms: empty and one-column slices, widths
around the four columns a lane takes at once, more rows than a block has warps, rows of a wider
buffer, and lists on both sides of the size that goes through the device.  Values are copied:
equal bit for bit."""
import numpy as np
import pytest

from tests.conftest import has_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,widths", [(1, [0, 1, 31, 32, 33]), (9, [127, 128, 129, 0]), (60, [700] * 20), (16, [1023] * 64),
                                         (16, [1024] * 65)])
def test_slices_equal_the_columns(rows, widths):
    if not has_gpu():
        pytest.skip("no CUDA device")
    import torch
    from seticore_b200.dedoppler import gather_hit_slices
    rng = np.random.default_rng(rows + len(widths))
    N = 5001
    x = rng.standard_normal((rows + 2, N + 7)).astype(np.float32)
    view = torch.from_numpy(x).cuda()[:, 3:3 + N]
    bounds = []
    for w in widths:
        b = int(rng.integers(0, N - w + 1))
        bounds.append((b, b + w))
    for stream in (None, torch.cuda.Stream()):
        if stream is not None:
            stream.wait_stream(torch.cuda.current_stream())
        got = gather_hit_slices(view, rows, N, bounds, stream=stream)
        assert len(got) == len(bounds)
        for g, (b, e) in zip(got, bounds):
            np.testing.assert_array_equal(g, x[:rows, 3 + b:3 + e])
