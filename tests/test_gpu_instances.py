"""Each kernel instance by itself against the oracle: no hand-over, which would
move most traces of a small batch to the 512-thread instance before their first
pass.  The edge inputs of the spline solve and the evaluation (short and long
systems, wide right-hand sides, zero couplings, plateaus, -0) and the golden
groups, on both time axes, both types and every knot placement that a small
arena forces; and spacings on both sides of the longest one that the integer
axis's quotients take."""
import hashlib
import os

import numpy as np
import pytest

import cases
from test_gpu_envelopes import _traces as edge_traces
from test_gpu_f32_rows import _traces as f32_traces

pytestmark = pytest.mark.gpu


def _launcher(variant, arena=0, **cfg):
    from cuda_emd import EMDKernelConfig
    L = EMDKernelConfig(**cfg).build()
    L._plan.set_variant(variant)
    L._plan.set_arena(arena)
    L._plan.set_tail(0)
    return L


def _run(L, X, T):
    import torch
    out = [o.cpu().numpy() for o in L.run(torch.from_numpy(X).cuda(),
                                          None if T is None else torch.from_numpy(T).cuda())]
    L.check_status()
    return out


def _compare(L, X, T, real, **cfg):
    from oracle import emd_oracle as O
    dt = np.float32 if real == "float" else np.float64
    Tx = np.arange(X.shape[1], dtype=dt) if T is None else T
    got = _run(L, X, T)
    for i, x in enumerate(X):
        with np.errstate(all="ignore"):
            r = O.emd_signal(x, Tx, O.OracleConfig(real_t=real, **cfg))
        assert (int(got[1][i]), int(got[2][i])) == (r.n_imfs, r.overflow), i
        assert got[0][i].tobytes() == r.imfs.astype(dt).tobytes(), i


VARIANTS = [("double", 4), ("double", 5), ("double", 6), ("double", 2),
            ("float", 4), ("float", 5), ("float", 6), ("float", 2)]


@pytest.mark.parametrize("real,variant", VARIANTS)
@pytest.mark.parametrize("axis", ["arange", "given"])
@pytest.mark.parametrize("nbsym", [2, 3])
def test_edge_inputs(real, variant, axis, nbsym):
    dt = np.float32 if real == "float" else np.float64
    with np.errstate(over="ignore"):
        X = edge_traces().astype(dt)
    if real == "float":
        X = X[np.isfinite(X).all(1) & (np.abs(X).max(1) < 2.0 ** 60)]
    T = None if axis == "arange" else np.cumsum(
        np.random.default_rng(3).uniform(1.0, 3.0, size=X.shape[1])).astype(dt)
    cfg = dict(max_iteration=12, max_imfs=6, nbsym=nbsym)
    _compare(_launcher(variant, real_t=real, **cfg), X, T, real, **cfg)


@pytest.mark.parametrize("variant", [4, 5, 6, 2])
@pytest.mark.parametrize("axis", ["arange", "given"])
def test_unusual_float_rows(variant, axis):
    X = np.stack(f32_traces()).astype(np.float32)
    T = None if axis == "arange" else np.arange(X.shape[1], dtype=np.float32)
    cfg = dict(max_iteration=6, max_imfs=4)
    _compare(_launcher(variant, real_t="float", **cfg), X, T, "float", **cfg)


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("room", [0, 800, 9000, 15000, 21000])
def test_every_placement(real, room):
    """A 128-thread CTA's arena from a trace's fixed part upwards: between them
    these traces take every knot placement on their first pass."""
    from cuda_emd import _native
    from oracle import emd_oracle as O
    dt = np.float32 if real == "float" else np.float64
    X = edge_traces()[[10, 13, 16, 31, 33]]
    n = X.shape[1]
    cfg = dict(max_iteration=8, max_imfs=5)
    L = _launcher(4, real_t=real, **cfg)
    fixed = L._plan.min_arena(n)
    if real == "double":
        first = [O.find_extrema(x) for x in X]
        taken = {_native.pass_placement(L.config.to_c(), n, fixed + r, e.ind_max.size, e.ind_min.size)
                 for e in first for r in (0, 800, 9000, 15000, 21000)}
        assert taken == {0, 1, 2, 3, 4, 5}
        L._plan.set_arena(fixed + room)
    else:                                      # half the proto-IMF, lanes and knots
        L._plan.set_arena(fixed - 4 * n - 3072 + 32 + room // 2)
    _compare(L, X.astype(dt), None, real, **cfg)


@pytest.mark.parametrize("real,variant", [("double", 2), ("double", 4), ("float", 2), ("float", 5)])
def test_golden_groups(golden, real, variant):
    here = os.path.dirname(os.path.abspath(__file__))
    g = golden if real == "double" else np.load(os.path.join(here, "golden", "ref_golden_f32.npz"))
    for name in (c["name"] for c in cases.groups()):
        X, T = g[f"{name}__signals"], g[f"{name}__T"]
        c = [int(v) for v in g[f"{name}__cfg"]]
        cfg = dict(zip(("max_extrema", "nbsym", "max_iteration", "max_imfs"), c))
        L = _launcher(variant, real_t=real, **cfg)
        for Tx in ([T, None] if np.array_equal(T, np.arange(X.shape[1])) else [T]):
            imfs, n_imfs, ovf = _run(L, X, Tx)[:3]
            for b in range(X.shape[0]):
                assert n_imfs[b] == g[f"{name}__nofma__n_imfs"][b], (name, b)
                sha = hashlib.sha256(imfs[b].tobytes()).hexdigest().encode()
                assert sha == g[f"{name}__nofma__sha"][b], (name, b)


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("gap", [65535, 65536, 65537])
def test_longest_integer_spacing(real, gap):
    """One pair of neighbouring maxima `gap` apart: up to 65536 the integer
    axis's quotients, beyond it the search and the division."""
    dt = np.float32 if real == "float" else np.float64
    n, at = 131000, 30000
    k = np.r_[np.arange(10, at, 1000), at, at + gap // 2, at + gap, np.arange(at + gap + 700, n - 10, 900)]
    v = np.where((np.arange(k.size) - np.searchsorted(k, at)) % 2 == 0, 1.0, -1.0)
    v = v * (1.0 + 0.2 * np.cos(np.arange(k.size)))
    x = np.interp(np.arange(n), np.r_[0, k, n - 1], np.r_[0.1, v, 0.1]).astype(dt)
    from oracle import emd_oracle as O
    e = O.find_extrema(x)
    assert np.diff(e.ind_max).max() == gap and np.diff(e.ind_min).max() < 65535
    cfg = dict(max_iteration=2, max_imfs=3)
    _compare(_launcher(1, real_t=real, **cfg), x[None], None, real, **cfg)
