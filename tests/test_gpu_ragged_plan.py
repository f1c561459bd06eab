"""The ragged runner on buffers that are refilled with other lengths: the plan
follows the lengths (a trace longer than its stale tier would come out flagged
and empty), with and without a graph; and the one call that cannot look at
them, a stream capture, takes the plan made just before it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(lens, seed):
    from cuda_emd import workloads as W
    return (np.concatenate([W.sinusoid_batch(1, int(n), seed=seed + k)[0] for k, n in enumerate(lens)]),
            np.r_[0, np.cumsum(lens)].astype(np.int64))


LENS = [300, 7000, 500, 900, 2500, 400]


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("host", [False, True])
def test_refilled_buffers(graph, host):
    import torch
    from cuda_emd import EMDKernelConfig
    from cuda_emd.ragged import RaggedRunner
    batches = [_batch(LENS, 5), _batch(LENS[::-1], 50), _batch(sorted(LENS), 90), _batch(LENS, 5)]
    v = torch.empty(batches[0][0].shape[0], dtype=torch.float64, device="cuda")
    o = torch.empty(len(LENS) + 1, dtype=torch.int64, device="cuda")
    runner = RaggedRunner(cache_path=None, autotune=False)
    outs = runner._alloc_out(v, o)
    for vals, offs in batches:
        v.copy_(torch.from_numpy(vals))
        o.copy_(torch.from_numpy(offs))
        got = runner.run(v, o, outs=outs, use_graph=graph, offsets_host=offs if host else None)
        ref = EMDKernelConfig().build().run_ragged(v, o)
        runner.check_status()
        for a, b in zip(ref, got):
            assert torch.equal(a, b)


def test_capture_takes_the_plan_made_before_it():
    import torch
    from cuda_emd.ragged import RaggedRunner
    vals, offs = _batch(LENS, 5)
    v, o = torch.from_numpy(vals).cuda(), torch.from_numpy(offs).cuda()
    runner = RaggedRunner(cache_path=None, autotune=False)
    ref = [x.clone() for x in runner.run(v, o)]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = runner.run(v, o)
    g.replay()
    torch.cuda.synchronize()
    for a, b in zip(ref, out):
        assert torch.equal(a, b)
