"""Tail migration from the 256-thread instance and over the host pipeline's
input groups: the same bits as without it, for a few and for all traces handed
over, dense and ragged, FP64 and FP32, both time axes, and batches of one to
many groups."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _launcher(variant, tail, real="double"):
    from cuda_emd import EMDKernelConfig
    L = EMDKernelConfig(real_t=real).build()
    if variant:
        L._plan.set_variant(variant)
    L._plan.set_tail(tail)
    return L


def _np(out):
    return [o.cpu().numpy() if hasattr(o, "cpu") else np.asarray(o) for o in out]


def _same(a, b):
    for x, y in zip(a, b):
        assert x.dtype == y.dtype and np.array_equal(x, y)


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("axis", [False, True])
def test_half_wide_hand_over(real, axis):
    import torch
    from cuda_emd import workloads as W
    dt = np.float32 if real == "float" else np.float64
    rng = np.random.default_rng(3)
    n = 2600
    X = np.concatenate([W.seismic_batch(330, n, seed=4), W.sinusoid_batch(60, n, seed=5),
                        np.stack([W.chirp_trace(rng, n) for _ in range(4)])]).astype(dt)
    T = torch.arange(n, device="cuda").to(torch.float64 if real == "double" else torch.float32)
    x = torch.from_numpy(X).cuda()
    ref = _np(_launcher(2, 0, real).run(x, T if axis else None))
    for tail in (-1, 40, 1 << 30):
        _same(ref, _np(_launcher(2, tail, real).run(x, T if axis else None)))


def test_half_wide_hand_over_ragged():
    import torch
    from cuda_emd import workloads as W
    vals, offs, _ = W.ragged_mix(500, lo=200, hi=4000, seed=6)
    v, o = torch.from_numpy(vals).cuda(), torch.from_numpy(offs).cuda()
    ref = _np(_launcher(2, 0).run_ragged(v, o))
    for tail in (-1, 1 << 30):
        _same(ref, _np(_launcher(2, tail).run_ragged(v, o)))


@pytest.mark.parametrize("batch,n", [(1, 700), (63, 700), (200, 2048), (1100, 1000), (2600, 512), (1300, 2500)])
def test_host_pipeline_hands_over_across_its_groups(batch, n):
    from cuda_emd import workloads as W
    X = W.seismic_batch(batch, n, seed=7) if batch < 300 else np.tile(
        W.seismic_batch(130, n, seed=7), (batch // 130 + 1, 1))[:batch]
    L = _launcher(0, 0)
    ref = _np(L.run_host(X, None))
    T = np.arange(n, dtype=np.float64)
    for tail in (-1, 1 << 30):
        M = _launcher(0, tail)
        _same(ref, _np(M.run_host(X, None)))
        _same(ref, _np(M.run_host(X, T)))            # again, on the same plan
