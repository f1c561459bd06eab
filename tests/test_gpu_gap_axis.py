"""Given time axes whose spacings lie far apart (a gap in the record, of any
length): the rows' quotients are tested then, the evaluation's are not as long
as every spacing is in [2^-100, 2^100).  Both sides of either line, every
instance, against the oracle."""
import numpy as np
import pytest

from test_gpu_envelopes import _zigzag

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [4, 2, 1])
@pytest.mark.parametrize("gap", [11.0, 12.9, 24.0, 38.0, 46.0])
@pytest.mark.parametrize("unit", [0.0, -90.0, -101.5, 60.0])
def test_axis_with_a_gap_equals_the_oracle(variant, gap, unit):
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    rng = np.random.default_rng(int(10 * gap))
    n = 600
    X = np.stack([_zigzag(rng, n, k) for k in (9, 40, 66, 150)] + [rng.normal(size=n)])
    step = rng.uniform(1.0, 1.5, size=n - 1)
    step[250] = 2.0 ** gap
    # the gap is short enough for every mirrored knot to keep a position of its own
    T = np.concatenate([np.cumsum(step[:250][::-1])[::-1] * -1.0, [0.0],
                        step[250] + np.r_[0.0, np.cumsum(step[251:])]]) * 2.0 ** unit
    assert (np.diff(T) > 0).all()
    cfg = dict(max_iteration=6, max_imfs=4)
    L = EMDKernelConfig(**cfg).build()
    L._plan.set_variant(variant)
    L._plan.set_tail(0)
    got = [o.cpu().numpy() for o in L.run(torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda())]
    for i in range(X.shape[0]):
        with np.errstate(all="ignore"):
            r = O.emd_signal(X[i], T, O.OracleConfig(**cfg))
        assert int(got[1][i]) == r.n_imfs, i
        same = (got[0][i].view(np.int64) == r.imfs.view(np.int64)) | (np.isnan(got[0][i]) & np.isnan(r.imfs))
        assert same.all(), (i, int((~same).sum()))
