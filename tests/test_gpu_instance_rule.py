"""Which kernel instance a plan takes for a trace length changes no bit: both
sides of each line of the rule, against the 128-thread instance without tail
migration, on both time axes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(X, T, real, variant=0, tail=-1):
    import torch
    from cuda_emd import EMDKernelConfig
    dt = np.float32 if real == "float" else np.float64
    L = EMDKernelConfig(real_t=real, max_iteration=40).build()
    if variant:
        L._plan.set_variant(variant)
    L._plan.set_tail(tail)
    return [o.cpu().numpy() for o in L.run(torch.from_numpy(X.astype(dt)).cuda(),
                                           torch.arange(X.shape[1], device="cuda").to(
                                               torch.from_numpy(X.astype(dt)[:1, :1]).dtype)
                                           if T else None)]


@pytest.mark.parametrize("axis", [False, True])
@pytest.mark.parametrize("real,n", [("double", 2048), ("double", 2049), ("double", 4096), ("double", 4097),
                                    ("float", 2048), ("float", 2049),
                                    ("float", 4096), ("float", 4097), ("float", 16384),
                                    ("float", 16385)])
def test_rule_changes_no_bit(real, n, axis):
    from cuda_emd import workloads as W
    X = np.tile(np.concatenate([W.seismic_batch(20, n, seed=11), W.sinusoid_batch(3, n, seed=12)]),
                (14, 1))[:310]
    ref = _run(X[:23], axis, real, variant=4, tail=0)
    for a, b in zip(ref, _run(X, axis, real)):
        for k in range(0, 299, 23):
            m = min(23, len(X) - k)
            assert np.array_equal(a[:m], b[k:k + m]), k


@pytest.mark.parametrize("axis", [False, True])
@pytest.mark.parametrize("tail", [-1, 200, 1 << 30])
def test_five_float_ctas_hand_over(tail, axis):
    from cuda_emd import workloads as W
    X = np.concatenate([W.seismic_batch(800, 600, seed=13), W.sinusoid_batch(100, 600, seed=14)])
    for a, b in zip(_run(X, axis, "float", 5, 0), _run(X, axis, "float", 5, tail)):
        assert np.array_equal(a, b)
