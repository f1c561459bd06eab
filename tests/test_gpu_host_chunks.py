"""The host pipeline's copy-back chunks: 8 to 64 traces by the rows' size, the last
chunk and the last group short, against the device path, on a plan that is used
for several sizes in turn."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# samples -> traces a chunk: 100 -> 64, 256 -> 64, 300 -> 54, 700 -> 23, 2047 / 2048 -> 8
SIZES = [(70, 100), (64, 256), (109, 300), (1030, 300), (1100, 700), (9, 2047), (1025, 2048), (5000, 33), (3, 1)]


def test_host_batches_equal_the_device_path():
    import torch
    from cuda_emd import EMDKernelConfig, workloads as W
    L, D = EMDKernelConfig().build(), EMDKernelConfig().build()
    for batch, n in SIZES + SIZES[:3]:
        X = np.tile(W.sinusoid_batch(min(batch, 90), n, seed=n), (batch // 90 + 1, 1))[:batch].copy()
        X *= np.linspace(1.0, 2.0, batch)[:, None]
        host = L.run_host(X, None)
        dev = [o.cpu().numpy() for o in D.run(torch.from_numpy(X).cuda(), None)]
        for a, b in zip(host, dev):
            assert np.array_equal(np.asarray(a), b), (batch, n)
