"""The packed strip code (both halves of the Taylor tree in float2 adds), executed on the CPU: each
generated function is translated line by line into Python, run on random float32 rows and
compared bit for bit with the recursion of taylor.h:30-86 inside the sheared strip, as
test_generator.py does for the single-float forms."""
import re

import numpy as np
import pytest

from tests.test_generator import _reference, _rows, gen


class Pair:
    __slots__ = ("x", "y")

    def __init__(self, x, y):
        self.x, self.y = np.float32(x), np.float32(y)


def _run(code, rows, S, emit):
    out, depth = [], 0
    for raw in code.splitlines():
        t = raw.strip().rstrip(";")
        if not t or t.startswith(("template", "__device__", "const Row", "#pragma", "taylor_")):
            continue
        m = re.match(r"for \(int it = 0; it < (\d+); \+\+it\) \{$", t)
        if m:
            out.append(f"for it in range({m.group(1)}):")
            depth = 1
            continue
        if t == "}":
            depth = 0
            continue
        t = re.sub(r"^float2? (\w+)\[(\d+)\]$", r"\1 = [None] * \2", t)
        t = re.sub(r"^const (?:float2|float|int) ", "", t).replace("0.0f", "F0")
        t = re.sub(r"^fold\(mrow, ", "fold(", t)
        out.append("    " * depth + t.replace("sink.put(", "put("))
    top, vals = [np.float32(0)] * S, {}

    class Row(list):  # a window: nothing left of it is read
        def __getitem__(self, j):
            assert j >= 0
            return list.__getitem__(self, j)

    def fold(i, v):
        top[i] = max(top[i], v)

    def put(i, c, v):
        vals[(i, c)] = v

    env = {"row": [Row(r) for r in rows], "F0": np.float32(0), "fmaxf": lambda a, b: a if a >= b else b,
           "fmax3": lambda a, b, c: max(a, b, c), "make_float2": Pair, "fold": fold, "put": put,
           "__fadd2_rn": lambda a, b: Pair(a.x + b.x, a.y + b.y)}
    exec(compile("\n".join(out), "<generated>", "exec"), env)
    return vals if emit else top


def _parts(configs):
    for R, nparts, U, IT in configs:
        for k in range(nparts):
            yield R, k * R // nparts, (k + 1) * R // nparts, U, IT


# the compiled forms, and longer strips of every row count (more than one loop iteration)
@pytest.mark.parametrize("cfg", list(_parts(gen.X2_CONFIGS + [(8, 1, 11, 3), (16, 1, 11, 3), (32, 2, 11, 2)])), ids=str)
def test_packed_form_equals_recursion(cfg):
    R, lo, hi, U, IT = cfg
    S = U * IT
    for seed in (1, 2):
        rows = _rows(R, S, seed)
        ref = _reference(rows, R, lo, hi, S)
        want = [max([np.float32(0)] + [ref[(i, p)] for i in range(hi - lo)]) for p in range(S)]
        got = _run(gen.gen_strip_x2(R, lo, hi, U, IT), rows, S, False)
        assert [np.float32(v).view(np.uint32) for v in got] == [np.float32(v).view(np.uint32) for v in want]


@pytest.mark.parametrize("cfg", list(_parts(gen.X2_EMIT_CONFIGS)), ids=str)
def test_packed_emitting_form_equals_recursion(cfg):
    R, lo, hi, U, IT = cfg
    S = U * IT
    rows = _rows(R, S, 3)
    ref = _reference(rows, R, lo, hi, S)
    got = _run(gen.gen_strip_x2(R, lo, hi, U, IT, emit=True), rows, S, True)
    assert got.keys() == ref.keys()
    assert all(np.float32(got[k]).view(np.uint32) == np.float32(ref[k]).view(np.uint32) for k in ref)
