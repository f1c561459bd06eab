"""The FP32 build on the integer time axis: its PCR and segment quotients are
formed without the division's tests, so the inputs here are those that make the
tests matter -- couplings below 2^-90, right-hand sides of -0, knots a few
samples or thousands apart, subnormal and very large traces.  Every bit must
equal the oracle's, and the given-axis build's, which divides."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 1400


def _pairs(n, gap, near=2):
    """Extrema in close pairs, far apart from one another."""
    x, at, k = np.zeros(n), [], 1
    while k < n - 1:
        at.append(k)
        k += near if len(at) % 4 else gap
    v = np.where(np.arange(len(at)) % 2 == 0, 1.0, -1.0) * (1.0 + 0.1 * np.cos(np.arange(len(at))))
    return np.interp(np.arange(n), at, v)


def _traces():
    t = np.arange(N, dtype=np.float64)
    rng = np.random.default_rng(17)
    mixed = np.sin(t * t / 700.0) + 0.3 * np.sin(t / 50.0) + 0.02 * rng.standard_normal(N)
    level = np.where(np.arange(N) % 2 == 0, 1.0, -1.0)
    flat = level.copy()
    flat[1::4] = -0.0
    flat[3::4] = 0.0
    return [mixed, level, flat, mixed * 2.0 ** -135, mixed * 2.0 ** 60, _pairs(N, 60), _pairs(N, 17, 1),
            np.sin(t * 0.9) * np.exp(-t / 30.0) + np.sin(t / 200.0)]


def _check(X, variant, **cfg):
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    T = np.arange(X.shape[1], dtype=np.float32)
    ref = [O.emd_signal(x, T, O.OracleConfig(real_t="float", **cfg)) for x in X]
    for axis in (None, torch.from_numpy(T).cuda()):
        L = EMDKernelConfig(real_t="float", **cfg).build()
        L._plan.set_variant(variant)
        got = [o.cpu().numpy() for o in L.run(torch.from_numpy(X).cuda(), axis)]
        for i, r in enumerate(ref):
            assert int(got[1][i]) == r.n_imfs, i
            assert got[0][i].tobytes() == r.imfs.astype(np.float32).tobytes(), i


@pytest.mark.parametrize("variant", [0, 4, 5, 2, 1])
def test_unusual_rows(variant):
    _check(np.stack(_traces()).astype(np.float32), variant, max_iteration=6, max_imfs=4)


@pytest.mark.parametrize("gap,near", [(13000, 2), (7000, 1)])
def test_couplings_that_vanish_before_the_last_level(gap, near):
    _check(_pairs(131000, gap, near)[None].astype(np.float32), 0, max_iteration=1, max_imfs=2)
