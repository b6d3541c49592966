"""gather_hit_slices takes the bounds as any integers: numpy's 32-bit ones (a column of a hit table) must
not wrap in the size of the output."""
import numpy as np
import pytest
import torch

from seticore_b200 import dedoppler


class _Stop(Exception):
    pass


@pytest.mark.parametrize("kind", [int, np.int32, np.int64])
def test_output_size_does_not_wrap(monkeypatch, kind):
    asked = []
    real = torch.empty

    def empty(size, **kw):
        if not asked and kw.get("dtype") == torch.int64:  # the table of offsets and bounds
            return real(size, dtype=torch.int64)
        asked.append((size, kw))
        raise _Stop

    class Input:
        device = "cuda"

    monkeypatch.setattr(torch, "empty", empty)
    T, w = 1024, 1 << 20
    bounds = [(kind(0), kind(w)), (kind(5), kind(w + 5)), (kind(0), kind(w)), (kind(9), kind(9))]
    with pytest.raises(_Stop):
        dedoppler.gather_hit_slices(Input(), T, 1 << 21, bounds)
    (size, kw), = asked
    assert size == 3 * T * w  # 3 * 2^30 floats, beyond 32 bits
    assert not kw.get("pin_memory")  # on the device, as every large output
