"""Batches of more than 256 rows: their searches run on the engine's side streams while the planes of
one drift block are small (one by one they take 1.5 times as long), with the single searches' hits.
"""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_TIME = """
import torch
from seticore_b200 import Dedopplerer
T, N, n = 2048, 1024, 8
foff, tsamp = 1e6 / 262144, 0.268435456
x = torch.rand((n, T, N), generator=torch.Generator("cuda").manual_seed(1), device="cuda")
dd = Dedopplerer(T, N, foff * 1e-6, tsamp)
ms = []
for _ in range(8):
    dd.search_batch_raw(list(x), [-1] * n, list(range(n)), 4.5 * foff / tsamp, 0.0, 16.0)
    ms.append(dd.last_stats().tree_ms)
print(min(ms[2:]))
"""


def _tree_ms(sides):
    env = dict(os.environ, SETICORE_B200_LEVEL_SIDES=str(sides), PYTHONPATH=ROOT)
    out = subprocess.run([sys.executable, "-c", _TIME], env=env, cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr[-2000:]
    return float(out.stdout.split()[-1])


@pytest.mark.gpu
def test_small_deep_searches_run_side_by_side():
    # Eight searches of 10 drift blocks, planes of 10 MB: level kernels of a few CTAs, one after another on
    # one stream and on four.  Measured 0.65 of the one-stream time; 0.85 leaves room for noise.
    assert _tree_ms(3) < 0.85 * _tree_ms(0)


@pytest.mark.gpu
@pytest.mark.parametrize("T,N", [(300, 1024), (512, 24576), (2048, 1024)])
def test_deep_batch_hits_equal_single_searches(T, N):
    import torch

    from seticore_b200 import Dedopplerer
    foff, tsamp, n = 1e6 / 262144, 0.268435456, 5
    md = 3.5 * foff / tsamp
    g = torch.Generator("cuda").manual_seed(T)
    xs = []
    for k in range(n):
        x = torch.empty((2048 if T > 1024 else 512, N), device="cuda").exponential_(generator=g)
        x[T:] = 0.0
        x[:T, 100 + 150 * k] += 2.0
        xs.append(x)
    key = lambda hits: [(h.index, h.drift_steps, h.power, h.snr) for h in hits]
    one = Dedopplerer(T, N, foff * 1e-6, tsamp)
    want = [key(one.search_raw(x, -1, 0, md, 0.0, 5.0)) for x in xs]
    dd = Dedopplerer(T, N, foff * 1e-6, tsamp)
    assert [key(h) for h in dd.search_batch_raw(xs, [-1] * n, list(range(n)), md, 0.0, 5.0)] == want
    assert len({w[0] for w in want}) == n  # every search has its own hits
