"""The dedoppler searches that a user of this package has it do, as cases that can be timed.

listed() and draw(rng) give the cases, prepare(case, seed) the inputs and the engine or pool that
a program keeps, run(state) one pass through the public entry points with its outputs, work(case)
the bytes and operations the pass cannot do without, and exact(case, seed) the outputs in 64 bits,
computed with torch and numpy alone.

Kinds of case:
  * "search": one coarse channel, Dedopplerer.search_raw; with "arrays" also the per-channel top
    path sums and column sums (Dedopplerer.channel_array);
  * "batch":  many coarse channels or beams of one shape, Dedopplerer.search_batch_raw;
  * "pool":   a mix of shapes, drift ranges and depths, SearchPool.search_raw;
  * "band":   one band of a multibeam buffer with an incoherent beam, multibeam.search_band;
  * "record": the device half of a file search: padding rows and DC spikes fixed in place
              (prepare_coarse_channels), the batch searched, and the columns around each hit
              gathered for the hit file (gather_hit_slices).

The power is Exp(1) noise times 1e9 under a slow bandpass, with linearly drifting tones well above
the threshold and broadband spikes, which is what a total-power filterbank holds; "integer" cases
hold the whole numbers of an 8-bit recording.
"""
import ctypes
import math

import numpy as np
import torch

from seticore_b200 import Dedopplerer, FilterbankMetadata, SearchPool, SearchRequest
from seticore_b200.dedoppler import gather_hit_slices, prepare_coarse_channels
from seticore_b200.multibeam import MultibeamBuffer, search_band

GBT_FOFF = 2.7939677       # Hz, the high spectral resolution product
GBT_TSAMP = 18.253611      # s
BEAM_FOFF = 1e6 / 262144   # Hz, beamformer output
BEAM_TSAMP = 0.268435456   # s


def _case(kind, T, N, **more):
    c = {"kind": kind, "T": T, "N": N, "foff": GBT_FOFF, "tsamp": GBT_TSAMP * 16 / max(T, 16), "max_drift": 4.0,
         "min_drift": 0.0, "snr": 16.0, "tones": 4, "spikes": 2}
    c.update(more)
    return c


def listed():
    return [
        # The smallest call: a narrow product searched as soon as it is there; launches and latency.
        _case("search", 16, 32768, name="coarse_16x32k", snr=14.0),
        # One coarse channel of a recording, with the spectra of top sums and column sums that a
        # viewer plots beside the hits.
        _case("search", 16, 1 << 20, name="coarse_16x1m", tones=8, arrays=True),
        # The same from an 8-bit recording: whole-number power, so many column sums are equal and
        # the statistics take the reference's own order.
        _case("search", 16, 1 << 20, name="coarse_8bit_16x1m", integer=True),
        # A ragged product: 60 timesteps (64 rounded), an odd channel count, and rows that are a
        # window of a wider buffer with an odd stride, so nothing is aligned.
        _case("search", 60, 100003, name="ragged_60x100003", pad=58, max_drift=10.0, min_drift=0.05, arrays=True),
        # A compute node's share of a wide band: the headline workload, and the largest.
        _case("batch", 16, 1 << 20, name="node_64x16x1m", count=64),
        # The same stored in 16 bits.
        _case("batch", 16, 1 << 20, name="node_bf16_32x16x1m", count=32, precision="bf16"),
        # 32-row recordings with the other coarse channel size that the file readers know.
        _case("batch", 32, 999424, name="rows32_8x32x999424", count=8),
        # Beamformer output: many rows, few drift blocks.
        _case("batch", 256, 131072, name="beams_32x256x128k", count=32, foff=BEAM_FOFF, tsamp=BEAM_TSAMP,
              max_drift=10.0),
        _case("batch", 256, 131072, name="beams_fp16_16x256x128k", count=16, foff=BEAM_FOFF, tsamp=BEAM_TSAMP,
              max_drift=10.0, precision="fp16"),
        # Requests of many users at once: uneven shapes and drift ranges in one pool call.
        _case("pool", 256, 1 << 20, name="uneven_24", count=24, mix=4000, spikes=0),
        # The beamforming pipeline's step: each coherent beam of a band, then the incoherent beam's
        # power along every hit.
        _case("band", 64, 32768, name="band_5x4x64x32k", beams=5, count=4, foff=BEAM_FOFF, tsamp=BEAM_TSAMP,
              max_drift=20.0),
        # A file search once its rows are on the device: 15 timesteps padded to 16, a DC spike in
        # each coarse channel, and a .hits file that keeps the columns around every hit.
        _case("record", 15, 1033216, name="record_8x15x1033216", count=8, dc_spike=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """A channel count: a power of two, a multiple of 16 or any number, spread over the logarithm."""
    n = _log_int(rng, lo, hi)
    how = rng.randrange(3)
    if how == 0:
        return 1 << max(1, round(math.log2(n)))
    return n // 16 * 16 if how == 1 else n


def draw(rng):
    top = work(_named("node_64x16x1m"))
    while True:
        kind = rng.choice(["search", "search", "search", "batch", "batch", "batch", "pool", "band", "record"])
        if kind == "pool":
            c = _case("pool", 256, 1 << 20, count=rng.randint(2, 24), mix=rng.randrange(1 << 30), spikes=0)
        elif kind == "band":
            c = _case("band", rng.choice([16, 32, 64, 128]), _size(rng, 8192, 1 << 17), beams=rng.randint(2, 6),
                      count=rng.randint(1, 6), foff=BEAM_FOFF, tsamp=BEAM_TSAMP, max_drift=rng.uniform(2.0, 20.0))
        elif kind == "record":
            c = _case("record", rng.choice([15, 16, 32, _log_int(rng, 4, 128)]), _size(rng, 1 << 15, 1 << 20),
                      count=_log_int(rng, 1, 32), dc_spike=rng.random() < 0.5, max_drift=rng.uniform(1.0, 10.0))
        else:
            T = rng.choice([16, 16, 32, 256, _log_int(rng, 4, 500)])
            if rng.random() < 0.3:
                foff, tsamp = BEAM_FOFF, BEAM_TSAMP
            else:
                foff, tsamp = GBT_FOFF, GBT_TSAMP * 16 / max(T, 16)
            c = _case(kind, T, _size(rng, 1 << 14, 1 << 20), foff=foff, tsamp=tsamp, max_drift=rng.uniform(1.0, 10.0),
                      min_drift=rng.choice([0.0, 0.05]), tones=rng.randint(1, 8), spikes=rng.randint(0, 2))
            if kind == "batch":
                c["count"] = _log_int(rng, 2, 64)
                if rng.random() < 0.4:
                    c["precision"] = rng.choice(["bf16", "fp16"])
            else:
                c["pad"] = rng.choice([0, 0, rng.randint(1, 64)])
                c["arrays"] = rng.random() < 0.5
                if rng.random() < 0.25:
                    c["integer"] = True
        w = work(c)
        if w["bytes"] <= top["bytes"] and w["flops"] <= top["flops"]:
            return c


def _named(name):
    return next(c for c in listed() if c["name"] == name)


# ---- shapes -------------------------------------------------------------------------------------

def _rounded(T):
    r = 1
    while r < T:
        r *= 2
    return r


def _plan(c):
    """(drift rate resolution Hz/s, first drift block, last, window size) of a search of this shape."""
    Tr = _rounded(c["T"])
    res = 1e6 * (c["foff"] * 1e-6) / ((Tr - 1) * c["tsamp"])
    nmax = c["max_drift"] / abs(res * (Tr - 1))
    return res, int(math.floor(-nmax)), int(math.floor(nmax)), int(2 * math.ceil(nmax * (Tr - 1)))


def _searches(c):
    """The single searches a case is made of (shape, drift range and threshold of each)."""
    if c["kind"] == "pool":
        rng = np.random.default_rng(c["mix"])
        out = []
        for _ in range(c["count"]):
            T = int(rng.choice([16, 32, 64, 128, 256]))
            N = int(rng.choice([65536, 131072, 262144, 1 << 20]))
            out.append(_case("search", T, N, max_drift=float(rng.uniform(1.0, 10.0)), tones=int(rng.integers(1, 7)),
                             spikes=0))
        return out
    if c["kind"] == "band":
        return [c] * ((c["beams"] - 1) * c["count"])
    return [c] * c.get("count", 1)


def work(case):
    """Bytes: the input read once (padding rows too, they are part of the buffer), the hits and the
    returned arrays written once.  Operations: one add for each distinct partial sum of the Taylor tree -- blocks of L rows
    have ndb * (L - 1) + 1 distinct drifts, those of neighbouring drift blocks meeting at their
    ends -- and one for each column sum term."""
    nbytes = flops = 0.0
    for s in _searches(case):
        Tr, N = _rounded(s["T"]), s["N"]
        _, dmin, dmax, _ = _plan(s)
        ndb = dmax - dmin + 1
        adds, L = Tr, 2
        while L <= Tr:
            adds += (Tr // L) * (ndb * (L - 1) + 1)
            L *= 2
        flops += float(adds) * N
        nbytes += 4.0 * Tr * N + 40.0 * (s["tones"] + s["spikes"])
        if case.get("arrays"):
            nbytes += 8.0 * N
    return {"bytes": nbytes, "flops": flops}


# ---- inputs -------------------------------------------------------------------------------------

def _power(c, seed, out):
    """Fills out ([rounded T][N], zeros past T) with noise, tones and spikes."""
    T, N = c["T"], c["N"]
    g = torch.Generator(device=out.device)
    g.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    out[T:].zero_()
    x = torch.linspace(0.0, 1.0, N, device=out.device)
    a, b, d = rng.normal(size=3)
    shape = a * x + b * x * x + d * x ** 3
    band = 1.0 + 0.1 * shape / shape.abs().max().clamp_min(1e-6)
    body = out[:T]
    scale = 12.0 if c.get("integer") else 1e9
    if body.is_contiguous():
        body.exponential_(1.0, generator=g)
    else:
        body.copy_(torch.empty((T, N), device=out.device).exponential_(1.0, generator=g))
    body.mul_(band).mul_(scale)
    _, dmin, dmax, _ = _plan(c)
    reach = min(N // 4, (max(-dmin, dmax) + 1) * T + 8)
    rows, cols, vals = [], [], []
    t = np.arange(T)
    for k in range(c["tones"] + c["spikes"]):
        amp = (rng.uniform(25.0, 100.0) if k < c["tones"] else 50.0) * scale * math.sqrt(T) / T
        lim = min(c["max_drift"], 4.0)
        rate = rng.uniform(-lim, lim) if k < c["tones"] else 0.0
        col = int(rng.integers(reach, N - reach)) + np.round(rate * t * c["tsamp"] / c["foff"]).astype(np.int64)
        ok = (col >= 0) & (col < N)
        rows.append(t[ok])
        cols.append(col[ok])
        vals.append(np.full(int(ok.sum()), amp, dtype=np.float32))
    if rows:
        at = [torch.from_numpy(np.concatenate(v)).to(out.device) for v in (rows, cols)]
        out.index_put_(tuple(at), torch.from_numpy(np.concatenate(vals)).to(out.device), accumulate=True)
    if c.get("integer"):
        body.round_().clamp_(0.0, 255.0)
    return out


def _inputs(case, seed):
    """One tensor per search, views of wider buffers where the case has them."""
    if case["kind"] == "band":
        Tr, N, B, C = _rounded(case["T"]), case["N"], case["beams"], case["count"]
        data = torch.empty((B, Tr, N * C), dtype=torch.float32, device="cuda")
        for b in range(B):
            for k in range(C):
                _power(dict(case, tones=0, spikes=0) if b == B - 1 else case, seed * 1000 + b * C + k,
                       data[b, :, k * N:(k + 1) * N])
        return data
    if case["kind"] == "pool":
        blocks = [torch.empty((_rounded(s["T"]), s["N"]), dtype=torch.float32, device="cuda") for s in _searches(case)]
    else:
        blocks = _block(case).unbind(0)
    pad = case.get("pad", 0) // 2
    return [_power(s, seed * 1000 + k, b[:, pad:pad + s["N"]]) for k, (s, b) in enumerate(zip(_searches(case), blocks))]


def _block(case):
    """[search][row][channel] memory of searches of one shape, rows as long as the buffer they lie in."""
    return torch.empty((len(_searches(case)), _rounded(case["T"]), case["N"] + case.get("pad", 0)), dtype=torch.float32,
                       device="cuda")


def prepare(case, seed):
    st = {"case": case}
    foff = case["foff"] * 1e-6
    x = _inputs(case, seed)
    if case["kind"] == "pool":
        st["requests"] = [SearchRequest(t, s["T"], foff, s["tsamp"], s["max_drift"], s["min_drift"], s["snr"],
                                        precision=s.get("precision", "fp32"))
                          for t, s in zip(x, _searches(case))]
        st["pool"] = SearchPool()
        return st
    st["engine"] = Dedopplerer(case["T"], case["N"], foff, case["tsamp"])
    if case["kind"] == "band":
        st["buffer"] = MultibeamBuffer(case["beams"], _rounded(case["T"]), case["N"] * case["count"], data=x)
        beams = case["beams"] - 1  # the last one is incoherent
        st["metadata"] = FilterbankMetadata(
            fch1=8000.0, foff=foff, tsamp=case["tsamp"], coarse_channel_size=case["N"], num_timesteps=case["T"],
            num_channels=case["N"] * case["count"], num_coarse_channels=case["count"],
            source_names=["beam%d" % b for b in range(beams)], ras=[1.0] * beams, decs=[2.0] * beams)
        return st
    if case.get("precision"):
        st["engine"].set_precision(case["precision"])
    st["inputs"] = x
    if case["kind"] == "record":
        st["block"] = x[0].as_strided((len(x),) + tuple(x[0].shape), (x[0].numel(),) + tuple(x[0].stride()))
    return st


# ---- one pass -----------------------------------------------------------------------------------

def _table(case, values, dtype):
    """One column of the hit table: the hits' values, then zeros up to 256 rows per search (a table
    that holds more hits grows)."""
    out = np.zeros(max(256 * len(_searches(case)), len(values)), dtype=dtype)
    out[:len(values)] = values
    return out


def _records(case, lists):
    """The hit records of raw calls as a table (each search's lie one after another in memory)."""
    got = {"counts": np.array([len(h) for h in lists], dtype=np.int64)}
    full = [np.ctypeslib.as_array((type(h[0]) * len(h)).from_address(ctypes.addressof(h[0]))) for h in lists if len(h)]
    full = np.concatenate(full) if full else None
    for name, dtype in (("index", np.int32), ("drift_steps", np.int32), ("drift_rate", np.float64),
                        ("snr", np.float32), ("power", np.float32)):
        got[name] = _table(case, full[name] if full is not None else [], dtype)
    return got


def _columns(case, index, steps):
    """The columns kept with a hit: 40 either side of its path."""
    return max(min(index, index + steps) - 40, 0), min(max(index, index + steps) + 40, case["N"])


def _slice_table(case, slices):
    """The slices one after another, then zeros up to 2^16 values per search."""
    flat = np.concatenate([s.reshape(-1) for s in slices]) if slices else np.zeros(0, dtype=np.float32)
    out = np.zeros(max(len(_searches(case)) << 16, flat.size), dtype=flat.dtype)
    out[:flat.size] = flat
    return out


def _hits(case, hits):
    got = {"count": len(hits)}
    for name, dtype in (("index", np.int32), ("drift_steps", np.int32), ("coarse_channel", np.int32),
                        ("frequency", np.float64), ("drift_rate", np.float64), ("snr", np.float32),
                        ("power", np.float32), ("incoherent_power", np.float32)):
        got[name] = _table(case, [getattr(h, name) for h in hits], dtype)
    return got


def run(state):
    c = state["case"]
    if c["kind"] == "search":
        out = _records(c, [state["engine"].search_raw(state["inputs"][0], -1, 0, c["max_drift"], c["min_drift"], c["snr"])])
        if c.get("arrays"):
            out["top"] = state["engine"].channel_array("top")
            out["colsum"] = state["engine"].channel_array("colsum")
        return out
    if c["kind"] == "batch":
        n = len(state["inputs"])
        return _records(c, state["engine"].search_batch_raw(state["inputs"], [-1] * n, list(range(n)), c["max_drift"],
                                                            c["min_drift"], c["snr"]))
    if c["kind"] == "pool":
        return _records(c, state["pool"].search_raw(state["requests"]))
    if c["kind"] == "band":
        return _hits(c, search_band(state["engine"], state["buffer"], state["metadata"], 0, c["count"], c["max_drift"],
                                    c["snr"]))
    x = state["inputs"]
    prepare_coarse_channels(state["block"], c["T"], c["dc_spike"])
    lists = state["engine"].search_batch(x, None, [-1] * len(x), list(range(len(x))), c["max_drift"], c["min_drift"],
                                         c["snr"])
    slices = []
    for t, hits in zip(x, lists):
        slices += gather_hit_slices(t, c["T"], c["N"], [_columns(c, h.index, h.drift_steps) for h in hits])
    out = _hits(c, [h for hits in lists for h in hits])
    out["slices"] = _slice_table(c, slices)
    return out


# ---- the same in 64 bits ------------------------------------------------------------------------

def _tops(x, dmin, dmax):
    """The largest path sum of each start channel (floored at 0) and the first path that has it."""
    Tr, N = x.shape
    top = torch.zeros(N, dtype=torch.float64, device=x.device)
    path = torch.zeros(N, dtype=torch.int64, device=x.device)
    chan = torch.arange(N, device=x.device)
    for db in range(dmin, dmax + 1):
        cur = x.unsqueeze(1)  # [block][offset][start channel]
        M = 1
        while M < Tr:
            nxt = torch.empty((cur.shape[0] // 2, 2 * M, N), dtype=torch.float64, device=x.device)
            for off in range(2 * M):
                left, right = cur[0::2, off >> 1], cur[1::2, off >> 1]
                s = M * db + ((off + 1) >> 1)
                o = nxt[:, off]
                if abs(s) >= N:
                    o.copy_(left)
                elif s >= 0:
                    torch.add(left[:, :N - s], right[:, s:], out=o[:, :N - s])
                    o[:, N - s:] = left[:, N - s:]
                else:
                    torch.add(left[:, -s:], right[:, :s], out=o[:, -s:])
                    o[:, :-s] = left[:, :-s]
            cur, M = nxt, 2 * M
        last = chan + (Tr - 1) * db
        for off in range(Tr):
            better = (cur[0, off] > top) & (last >= 0) & (last + off < N)
            top = torch.where(better, cur[0, off], top)
            path = torch.where(better, torch.full_like(path, db * (Tr - 1) + off), path)
    return top, path


def _search64(c, x):
    """(index, drift steps, drift rate, snr, power) of the hits, and the top and column sums."""
    N = c["N"]
    res, dmin, dmax, w = _plan(c)
    x = x.double()
    top, path = _tops(x, dmin, dmax)
    colsum = x.sum(0)
    s = torch.sort(colsum).values
    median = float(s[N // 2])
    mid = s[int(math.ceil(0.05 * N)):int(math.floor(0.95 * N)) + 1]
    std = float(((mid - mid.mean()) ** 2).mean().sqrt())
    threshold = c["snr"] * std + median
    v, p = top.cpu().numpy(), path.cpu().numpy()
    nwin = -(-N // w)
    padded = np.full(nwin * w, -1.0)
    padded[:N] = v
    first = padded.reshape(nwin, w).argmax(axis=1) + np.arange(nwin) * w
    hits = []
    for i in first[padded[first] > threshold]:
        if v[max(0, i - w + 1):i + w].max() > v[i]:
            continue
        rate = float(p[i]) * res
        if abs(rate) >= c["min_drift"]:
            hits.append((int(i), int(p[i]), rate, (v[i] - median) / std, v[i]))
    return hits, top, colsum


def _path_sum(x, index, steps):
    Tr = x.shape[0]
    db = math.floor(steps / (Tr - 1))

    def add(t, L, off, c):
        if L == 1:
            return float(x[t, c])
        half = L // 2
        return add(t, half, off >> 1, c) + add(t + half, half, off >> 1, c + half * db + ((off + 1) >> 1))

    return add(0, Tr, steps - db * (Tr - 1), index)


def exact(case, seed):
    col = lambda hits, k: _table(case, [h[k] for h in hits], np.float64)  # noqa: E731
    if case["kind"] in ("search", "batch", "pool"):
        hits = []
        for s, x in zip(_searches(case), _inputs(case, seed)):
            h, top, colsum = _search64(s, x)
            hits += h
        out = {"counts": None, "index": None, "drift_steps": None, "drift_rate": col(hits, 2), "snr": col(hits, 3),
               "power": col(hits, 4)}
        if case.get("arrays"):
            out.update(top=top, colsum=colsum)
        return out
    N = case["N"]
    hits, inc, slices = [], [], []
    x = _inputs(case, seed)
    for k in range(case["count"]):
        if case["kind"] == "band":
            mine = []
            for b in range(case["beams"] - 1):
                mine += _search64(case, x[b, :, k * N:(k + 1) * N])[0]
            mine.sort(key=lambda h: h[1])
            noise = x[-1, :, k * N:(k + 1) * N].double().cpu().numpy()
            inc += [_path_sum(noise, h[0], h[1]) for h in mine]
        else:
            v = x[k]
            if case["dc_spike"]:
                v[:, N // 2] = (v[:, N // 2 - 1] + v[:, N // 2 + 1]) / 2
            mine = _search64(case, v)[0]
            for h in mine:
                lo, hi = _columns(case, h[0], h[1])
                slices.append(v[:case["T"], lo:hi].double().cpu().numpy())
        hits += [h + ((8000.0 if case["kind"] == "band" else 0.0) + (k * N + h[0]) * (case["foff"] * 1e-6),) for h in mine]
    out = {"count": None, "index": None, "drift_steps": None, "coarse_channel": None, "frequency": col(hits, 5), "drift_rate": col(hits, 2),
           "snr": col(hits, 3), "power": col(hits, 4), "incoherent_power": _table(case, inc, np.float64)}
    if case["kind"] == "record":
        out["slices"] = _slice_table(case, slices)
    return out
