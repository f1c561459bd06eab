"""Performance cases: what a user of this framework has it do, through its public entry points.

A case is a plain dict.  ``call`` names the entry point, the other fields the
size and the kind of trace:

  device    GPUBatchEMD on a CUDA batch [batch, n], T = arange
  axis      the same with a non-uniform time axis T
  float     the same with EMDKernelConfig(real_t="float")
  host      GPUBatchEMD on page-locked host memory, results into host buffers
  ragged    RaggedRunner on a CSR batch, lengths log-uniform in [lo, n]
  envelope  EMDBatchLauncher.run_envelope_only (extrema, mirroring, splines)

Kinds of trace: ``seismic`` (Ricker wavelets on random reflectivity plus
5-100 Hz noise at 10 dB, dt = 2 ms), ``tones`` (three tones, a trend, noise),
``slow`` (an oversampled record: the tones alone, at low frequencies, whose
extrema stay below max_extrema for tens of thousands of samples), ``mix``
(60 % seismic, 38 % tones, 2 % linear chirps).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.abspath("emd-cuda_b200"))

DT = 0.002
MAX_IMFS = 16

# Sift passes a trace takes on average (logged counts of these generators), for
# the operation count.  Noise-like traces past ~3,000 samples hold more extrema
# than max_extrema, and some of their IMFs run to the iteration cap.
PASSES = {"seismic": 65.0, "tones": 15.0, "slow": 23.0}
LONG_FROM = 2700
MAX_FLOPS = 1.4e11

_RUNNER = []


def listed():
    return [
        # one trace, an interactive look at a short record: latency only
        {"name": "one_trace_1024", "call": "device", "kind": "tones", "batch": 1, "n": 1024},
        # one shot gather of 3 s at 2 ms, fewer traces than the GPU has CTA slots
        {"name": "gather_96x1501", "call": "device", "kind": "seismic", "batch": 96, "n": 1501},
        # a monitoring window: many short smooth traces, round in decimal
        {"name": "tones_4096x1000", "call": "device", "kind": "tones", "batch": 4096, "n": 1000},
        # the equal-length production batch (the repository's head-to-head size)
        {"name": "seismic_16384x2048", "call": "device", "kind": "seismic", "batch": 16384, "n": 2048},
        # an irregularly sampled survey: its own time axis
        {"name": "axis_1024x1777", "call": "axis", "kind": "seismic", "batch": 1024, "n": 1777},
        # mid-length records
        {"name": "seismic_1024x4096", "call": "device", "kind": "seismic", "batch": 1024, "n": 4096},
        # long noisy records, past max_extrema
        {"name": "seismic_256x8192", "call": "device", "kind": "seismic", "batch": 256, "n": 8192},
        # a few very long oversampled records, longer than shared memory holds
        {"name": "slow_8x30011", "call": "device", "kind": "slow", "batch": 8, "n": 30011},
        # a batch that lives in host memory: copies, sift and copy-back
        {"name": "host_2048x2048", "call": "host", "kind": "seismic", "batch": 2048, "n": 2048},
        # the reference kernel's REAL_T = float
        {"name": "float_4096x1500", "call": "float", "kind": "seismic", "batch": 4096, "n": 1500},
        # mixed lengths through the tiered runner
        {"name": "ragged_2048x8192", "call": "ragged", "kind": "mix", "batch": 2048, "lo": 256, "n": 8192},
        # envelopes only, for inspection and quality control
        {"name": "envelope_4096x2048", "call": "envelope", "kind": "seismic", "batch": 4096, "n": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        call = rng.choice(["device", "device", "device", "device", "axis", "float", "host", "ragged", "envelope"])
        if call == "ragged":
            c = {"call": call, "kind": "mix", "lo": _log_int(rng, 200, 600), "n": _log_int(rng, 1500, 8192),
                 "batch": _log_int(rng, 512, 4096)}
        elif call == "envelope":
            kind = rng.choice(["seismic", "tones"])
            c = {"call": call, "kind": kind, "n": _log_int(rng, 200, 4096 if kind == "seismic" else 2500),
                 "batch": _log_int(rng, 64, 8192)}
        else:
            kind = rng.choice(["seismic", "seismic", "tones", "slow"])
            top = {"seismic": 6000, "tones": 2900, "slow": 32000}[kind]
            if call == "float":
                top = min(top, 2500)
            c = {"call": call, "kind": kind, "n": _log_int(rng, 300, top),
                 "batch": _log_int(rng, 64 if call in ("host", "float") else 1, 16384)}
        w = work(c)
        most = {"host": 1.5e8, "ragged": 3.0e9, "envelope": 1.0e9}.get(c["call"], 4.6e9)
        if w["flops"] <= MAX_FLOPS and w["bytes"] <= most:
            return c


# -- inputs -----------------------------------------------------------------

def _tones(g, b, n, kind):
    dev = "cuda"
    t = torch.arange(n, dtype=torch.float64, device=dev)
    if kind == "slow":
        lo, hi = (0.0005, 0.002, 0.006), (0.002, 0.006, 0.015)
    else:
        lo, hi = (0.005, 0.05, 0.15), (0.05, 0.15, 0.4)
    u = torch.rand((b, 10), generator=g, dtype=torch.float64, device=dev)
    x = (2e-3 * u[:, 9:10] - 1e-3) * t * (1.0 if kind == "tones" else 0.05)
    for k in range(3):
        f = lo[k] + (hi[k] - lo[k]) * u[:, k:k + 1]
        x += (0.5 + 1.5 * u[:, 3 + k:4 + k]) * torch.sin(2 * math.pi * (f * t + u[:, 6 + k:7 + k]))
    if kind == "tones":
        x += 0.05 * torch.randn((b, n), generator=g, dtype=torch.float64, device=dev)
    return x


def _seismic(g, b, n):
    dev = "cuda"
    out = torch.empty((b, n), dtype=torch.float64, device=dev)
    m = 1 << (n + 256).bit_length()                   # room past the end: no wrap-around
    f = torch.fft.rfftfreq(m, DT, dtype=torch.float64, device=dev)
    # 4th-order Butterworth band-pass magnitude, 5-100 Hz
    w = f.clamp(min=1e-6)
    band = 1.0 / torch.sqrt(1.0 + ((w * w - 500.0) / (w * 95.0)) ** 8)
    for s in range(0, b, 2048):
        k = min(2048, b - s)
        u = torch.rand((k, 2), generator=g, dtype=torch.float64, device=dev)
        peak = 10.0 + 50.0 * u[:, :1]
        spikes = 20 + (61 * u[:, 1:]).long()
        # one spike a layer, so that no two fall on one sample
        u = torch.rand((k, 80), generator=g, dtype=torch.float64, device=dev)
        layer = torch.arange(80, device=dev) + 0.5 * u
        pos = (n * layer / spikes).long().clamp(max=m - 1)
        v = torch.rand((k, 80), generator=g, dtype=torch.float64, device=dev) - 0.5
        amp = -torch.sign(v) * torch.log1p(-2.0 * v.abs().clamp(max=0.4999999))
        refl = torch.zeros((k, m + 80), dtype=torch.float64, device=dev)
        unused = torch.arange(80, device=dev) >= spikes
        pos = torch.where(unused, m + torch.arange(80, device=dev), pos)
        refl = refl.scatter_(1, pos, amp)[:, :m]
        # the Ricker wavelet's (zero-phase) spectrum
        q = (f / peak) ** 2
        sig = torch.fft.irfft(torch.fft.rfft(refl) * (q * torch.exp(-q)), n=m)[:, :n]
        noise = torch.randn((k, m), generator=g, dtype=torch.float64, device=dev)
        noise = torch.fft.irfft(torch.fft.rfft(noise) * band, n=m)[:, :n]
        ps = (sig * sig).mean(1, keepdim=True).clamp(min=1e-12)
        pn = (noise * noise).mean(1, keepdim=True)
        out[s:s + k] = sig + noise * torch.sqrt(ps / (10.0 * pn))
    return out


def _traces(kind, g, b, n):
    return _seismic(g, b, n) if kind == "seismic" else _tones(g, b, n, kind)


def _chirp(g, n):
    t = torch.arange(n, dtype=torch.float64, device="cuda")
    x = torch.sin(2 * math.pi * (0.001 * t + 0.5 * 0.449 * t * t / max(n - 1, 1)))
    return x + 0.01 * torch.randn(n, generator=g, dtype=torch.float64, device="cuda")


def _mix(case, g):
    rng = np.random.default_rng(case["batch"])        # the layout is the case's, the traces the seed's
    b, lo, hi = case["batch"], case["lo"], case["n"]
    lens = np.exp(rng.uniform(np.log(lo), np.log(hi), size=b)).astype(np.int64).clip(lo, hi)
    u = rng.uniform(size=b)
    offsets = np.zeros(b + 1, dtype=np.int64)
    np.cumsum(lens, out=offsets[1:])
    values = torch.empty(int(offsets[-1]), dtype=torch.float64, device="cuda")
    for i in range(0, b, 64):                         # each block of 64 from one padded batch
        at = range(i, min(i + 64, b))
        n = int(lens[i:i + 64].max())
        s, t = _seismic(g, len(at), n), _tones(g, len(at), n, "tones")
        for j, k in enumerate(at):
            m = int(lens[k])
            x = s[j, :m] if u[k] < 0.6 else t[j, :m] if u[k] < 0.98 else _chirp(g, m)
            values[int(offsets[k]):int(offsets[k + 1])] = x
    return values, torch.from_numpy(offsets).to("cuda")


def _axis(case, seed):
    rng = np.random.default_rng(seed + 1)
    return np.cumsum(rng.uniform(0.5, 1.5, size=case["n"]) * DT)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


# -- the calls ----------------------------------------------------------------

def prepare(case, seed):
    from cuda_emd import EMDKernelConfig, GPUBatchEMD
    g = _generator(seed)
    call, b, n = case["call"], case["batch"], case["n"]
    if call == "ragged":
        from cuda_emd.ragged import RaggedRunner
        values, offsets = _mix(case, g)
        # one runner per program, tuned on the batches it has seen
        if not _RUNNER:
            _RUNNER.append(RaggedRunner(cache_path=None))
        _RUNNER[0].run(values, offsets)
        return {"call": call, "runner": _RUNNER[0], "values": values, "offsets": offsets,
                "off_h": offsets.cpu().numpy()}
    x = _traces(case["kind"], g, b, n)
    if call == "envelope":
        return {"call": call, "launcher": EMDKernelConfig.for_device().build(), "x": x}
    if call == "float":
        emd = GPUBatchEMD(EMDKernelConfig.for_device(real_t="float"))
        x = x.float()
    else:
        emd = GPUBatchEMD()
    emd.warmup()
    state = {"call": call, "emd": emd, "x": x, "T": None, "out": None}
    if call == "axis":
        state["T"] = torch.from_numpy(_axis(case, seed)).cuda()
    if call == "host":
        state["x"] = x.cpu().pin_memory()
        state["out"] = (torch.empty((b, MAX_IMFS, n), dtype=torch.float64, pin_memory=True),
                        torch.empty(b, dtype=torch.int32, pin_memory=True),
                        torch.empty(b, dtype=torch.int32, pin_memory=True))
    return state


def run(state):
    call = state["call"]
    if call == "ragged":
        return state["runner"].run(state["values"], state["offsets"], offsets_host=state["off_h"])
    if call == "envelope":
        return state["launcher"].run_envelope_only(state["x"], None)
    emd = state["emd"]
    imfs, n_imfs, overflow = emd(state["x"], T=state["T"], out=state["out"])
    return imfs, n_imfs, overflow, emd.last_debug


def work(case):
    """Input once, output rows once; about 65 operations a sample and 20 a
    knot (a quarter of the samples, both envelopes) in each sift pass."""
    b, n = case["batch"], case["n"]
    if case["call"] == "ragged":
        n = (n - case["lo"]) / math.log(n / case["lo"])
    size = 4 if case["call"] == "float" else 8
    if case["call"] == "envelope":
        return {"bytes": b * (3.0 * n + 4.0 * 1028) * size, "flops": b * n * 60.0}
    if case["kind"] == "mix":
        passes = 135.0 * case["n"] / 8192.0
    else:
        passes = PASSES[case["kind"]]
        if case["kind"] == "seismic" and n > LONG_FROM:
            passes *= (n / LONG_FROM) ** 2.2
    return {"bytes": b * n * (1.0 + MAX_IMFS) * size, "flops": b * n * passes * 70.0}


# -- the same in plain numpy ----------------------------------------------------

def _extrema(s):
    d = np.diff(s)
    turn = d[:-1] * d[1:] < 0.0
    up = np.flatnonzero(turn & (d[:-1] > 0.0)) + 1
    down = np.flatnonzero(turn & (d[:-1] < 0.0)) + 1
    return up, down, int(np.count_nonzero(s[:-1] * s[1:] < 0.0))


def _mirror(t, s, up, down, nb=2):
    """Knots of both envelopes: true extrema with nb mirrored ones at each end."""
    n = len(s)

    def left(first, other, above):
        # `first`: the kind of extremum that comes first; `above`: it is the maxima
        over = s[0] > s[other[0]] if above else s[0] < s[other[0]]
        if over:
            return first[1:nb + 1][::-1], other[:nb][::-1], first[0]
        return first[:nb][::-1], np.append(other[:nb - 1][::-1], 0), 0

    def right(last, other, above):
        over = s[-1] > s[other[-1]] if above else s[-1] < s[other[-1]]
        if over:
            return last[-nb - 1:-1][::-1], other[-nb:][::-1], last[-1]
        return last[-nb:][::-1], np.append([n - 1], other[-(nb - 1):][::-1] if nb > 1 else []), n - 1

    if up[0] < down[0]:
        lu, ld, ls = left(up, down, True)
    else:
        ld, lu, ls = left(down, up, False)
    if up[-1] > down[-1]:
        ru, rd, rs = right(up, down, True)
    else:
        rd, ru, rs = right(down, up, False)
    lu, ld = (a if len(a) else b[:1] for a, b in ((lu, up), (ld, down)))
    ru, rd = (a if len(a) else b[-1:] for a, b in ((ru, up), (rd, down)))
    lu, ld, ru, rd = (np.asarray(a, dtype=np.int64) for a in (lu, ld, ru, rd))
    if max(2 * t[ls] - t[lu[0]], 2 * t[ls] - t[ld[0]]) > t[0]:
        if ls == up[0]:
            lu = up[:nb][::-1]
        else:
            ld = down[:nb][::-1]
        ls = 0
    if min(2 * t[rs] - t[ru[-1]], 2 * t[rs] - t[rd[-1]]) < t[-1]:
        if rs == up[-1]:
            ru = up[-nb:][::-1]
        else:
            rd = down[-nb:][::-1]
        rs = n - 1
    knots = []
    for a, mid, b in ((lu, up, ru), (ld, down, rd)):
        knots.append((np.concatenate([2 * t[ls] - t[a], t[mid], 2 * t[rs] - t[b]]),
                      np.concatenate([s[a], s[mid], s[b]])))
    return knots


def _spline(x, y, t):
    """Not-a-knot cubic spline through (x, y) at t."""
    n = len(x)
    if n <= 3:
        return np.polyval(np.polyfit(x - x[0], y, n - 1), t - x[0])
    h = np.diff(x)
    r = 6.0 * np.diff(np.diff(y) / h)
    a, b, c, d = h[:-1].copy(), 2.0 * (h[:-1] + h[1:]), h[1:].copy(), r.copy()
    a[0], b[0], c[0], d[0] = 0.0, h[0] + 2 * h[1], h[1] - h[0], h[1] * r[0] / (h[0] + h[1])
    a[-1], b[-1], c[-1], d[-1] = h[-2] - h[-1], 2 * h[-2] + h[-1], 0.0, h[-2] * r[-1] / (h[-2] + h[-1])
    k = np.arange(n - 2)
    s = 1
    while s < n - 2:                                  # cyclic reduction, all rows at once
        lo, hi = np.maximum(k - s, 0), np.minimum(k + s, n - 3)
        p, q = np.where(k >= s, a / b[lo], 0.0), np.where(k + s < n - 2, c / b[hi], 0.0)
        a, b, c, d = -p * a[lo], b - p * c[lo] - q * a[hi], -q * c[hi], d - p * d[lo] - q * d[hi]
        s *= 2
    m = np.empty(n)
    m[1:-1] = d / b
    m[0] = ((h[0] + h[1]) * m[1] - h[0] * m[2]) / h[1]
    m[-1] = ((h[-2] + h[-1]) * m[-2] - h[-1] * m[-3]) / h[-2]
    j = np.clip(np.searchsorted(x, t, side="right") - 1, 0, n - 2)
    p, q = (x[j + 1] - t) / h[j], (t - x[j]) / h[j]
    return p * y[j] + q * y[j + 1] + ((p ** 3 - p) * m[j] + (q ** 3 - q) * m[j + 1]) * h[j] ** 2 / 6.0


def _sift(x, t):
    """One trace's rows [16, n] and its IMF count."""
    rows = np.zeros((MAX_IMFS, len(x)))
    res, count, done = x.copy(), 0, False
    while not done and count < MAX_IMFS - 1:
        imf = res.copy()
        up, down, zeros = _extrema(imf)
        for _ in range(999):
            total = len(up) + len(down)
            if total <= 2 or not len(up) or not len(down):
                done = True
                break
            (ux, uy), (dx, dy) = _mirror(t, imf, up, down)
            old, imf = imf, imf - 0.5 * (_spline(ux, uy, t) + _spline(dx, dy, t))
            up, down, zeros = _extrema(imf)
            total = len(up) + len(down)
            step = ((imf - old) ** 2).sum()
            good = not ((uy < 0).any() or (dy > 0).any()) and (imf * imf).sum() >= 1e-10 and (
                step / (old.max() - old.min()) < 0.001 or (((imf - old) / imf) ** 2).sum() < 0.2
                or step / (old * old).sum() < 0.2)
            if good and abs(total - zeros) < 2:
                break
        rows[count] = imf
        res = res - imf
        count += 1
        done = done or res.max() - res.min() < 0.001 or np.abs(res).sum() < 0.005
    if total <= 2 and count > 0:
        count -= 1
        res = res + imf
    if np.abs(res).max() > 1e-8:
        rows[count] = res
        count += 1
    return rows, count


def exact(case, seed):
    """The envelopes, and the rows of small FP64 batches (each trace takes
    about 0.1 s here).  A float decomposition has no 64-bit counterpart: its
    stopping decisions are taken on float values."""
    b, n = case["batch"], case["n"]
    if case["call"] == "envelope":
        small = b * n <= 1.0e7
    else:
        small = case["call"] in ("device", "axis") and n <= 2500 and work(case)["flops"] <= 3.0e9
    if not small:
        return None
    x = _traces(case["kind"], _generator(seed), b, n).cpu().numpy()
    t = np.arange(n, dtype=np.float64)
    if case["call"] == "envelope":
        upper, lower = np.zeros((b, n)), np.zeros((b, n))
        for i in range(b):
            up, down, _ = _extrema(x[i])
            if len(up) + len(down) > 2 and len(up) and len(down):
                (ux, uy), (dx, dy) = _mirror(t, x[i], up, down)
                upper[i], lower[i] = _spline(ux, uy, t), _spline(dx, dy, t)
        return (upper, lower) + (None,) * 7
    if case["call"] == "axis":
        t = _axis(case, seed)
        t = (t - t[0]) / np.diff(t).min()
    rows, counts = zip(*(_sift(v, t) for v in x))
    return np.stack(rows), np.array(counts, dtype=np.int32), None, None
