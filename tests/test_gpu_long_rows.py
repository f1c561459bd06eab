"""Traces past 16,384 samples, where the zero-crossing count can fall back to the
reference's serial scan (a first sample of exactly zero, more than 64 extrema of
a kind in one of 128 chunks): rows whose residue is zero everywhere (the
iteration cap of one, a monotonic last row) right after a scan, first samples of
zero with and without such a chunk, on both sides of the line and with the
proto-IMF in global memory, bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traces(n):
    rng = np.random.default_rng(n)
    t = np.arange(n, dtype=np.float64)
    smooth = np.sin(t / 900.0) + 0.2 + 1e-4 * t          # ends in a monotonic row
    ramp = 0.5 + 1e-3 * t                                 # is one
    dense = rng.normal(size=n) + 0.01                     # more than 64 a chunk
    out = [smooth, ramp, dense]
    for x in (smooth, dense):
        z = x.copy()
        z[0] = 0.0
        out.append(z)
    z = np.sin(t / 700.0)                                 # starts at zero by itself
    z[2000:2400] += np.where(np.arange(400) % 2 == 0, 1.0, -1.0)
    out.append(z)
    return np.stack(out)


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("max_iteration", [1, 4])
@pytest.mark.parametrize("n", [16384, 16385, 20000, 30011])
def test_rows_after_a_scan_of_a_long_trace(n, max_iteration, real):
    import torch
    from cuda_emd import EMDKernelConfig
    from oracle import emd_oracle as O
    dt = np.float64 if real == "double" else np.float32
    X = _traces(n).astype(dt)
    cfg = dict(max_iteration=max_iteration, max_imfs=5)
    ref = [O.emd_signal(x, np.arange(n, dtype=dt), O.OracleConfig(real_t=real, **cfg)) for x in X]
    for variant in (4, 2, 1):
        L = EMDKernelConfig(real_t=real, **cfg).build()
        L._plan.set_variant(variant)
        L._plan.set_tail(0)
        for _ in range(3):
            imfs, n_imfs, ovf, dn, de, dz = (o.cpu().numpy() for o in L.run(
                torch.from_numpy(X).cuda(), None))
            for i, r in enumerate(ref):
                assert (int(n_imfs[i]), int(ovf[i])) == (r.n_imfs, r.overflow), (variant, i)
                assert np.array_equal(dn[i], r.debug_n) and np.array_equal(dz[i], r.debug_nzm), (variant, i)
                assert imfs[i].tobytes() == r.imfs.astype(dt).tobytes(), (variant, i)
