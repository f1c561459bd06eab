"""Tail migration and traces longer than the launch's announced maximum: a
128-thread CTA takes such a trace if its arena holds it (the wider instances
refuse it), and the continuation records, sized by that maximum, do not.  It
finishes where it is; every output equals the launch without hand-over, and
nothing is written past the records."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("variant", [0, 4])
def test_traces_longer_than_announced_stay(variant, real):
    import torch
    from cuda_emd import EMDKernelConfig, workloads as W
    dt = np.float32 if real == "float" else np.float64
    traces = [W.sinusoid_batch(1, n, seed=n)[0] for n in np.linspace(60, 200, 170).astype(int)]
    for k, n in ((5, 201), (50, 1500), (100, 3000), (160, 2500)):
        traces[k] = W.seismic_batch(1, n, seed=n)[0]
    offs = np.r_[0, np.cumsum([len(t) for t in traces])].astype(np.int64)
    v = torch.from_numpy(np.concatenate(traces).astype(dt)).cuda()
    o = torch.from_numpy(offs).cuda()

    def run(variant, tail, max_n):
        L = EMDKernelConfig(real_t=real).build()
        L._plan.set_variant(variant)
        L._plan.set_tail(tail)
        out = [x.cpu().numpy() for x in L.run_ragged(v, o, max_n=max_n)]
        L.check_status()
        return out

    ref = run(4, 0, 3000)
    for tail in (0, -1, 1 << 30):
        for a, b in zip(ref, run(variant, tail, 200)):
            assert np.array_equal(a, b), tail


def test_a_refused_trace_does_not_stop_the_hand_over():
    """A trace that no arena of the launch holds is flagged; the rest of the
    batch still hands its traces over.  Seen in the pass counters: on the
    512-thread instance, whose arena holds every knot of these traces, no pass
    spills, on the 128-thread one many do."""
    import torch
    from cuda_emd import EMDKernelConfig, workloads as W
    n = 2048
    X = W.seismic_batch(200, n, seed=21)

    def spilled(tail, long_one):
        traces = list(X)
        if long_one:
            traces.insert(7, np.cumsum(W.seismic_batch(1, 12000, seed=3)[0]))
        offs = np.r_[0, np.cumsum([len(t) for t in traces])].astype(np.int64)
        L = EMDKernelConfig().build()
        L._plan.set_variant(4)
        L._plan.set_tail(tail)
        L._plan.counters(reset=True)
        out = L.run_ragged(torch.from_numpy(np.concatenate(traces)).cuda(),
                           torch.from_numpy(offs).cuda(), max_n=n)
        n_imfs = out[1].cpu().numpy()
        if long_one:
            assert n_imfs[7] == 0
            with pytest.raises(ValueError):
                L.check_status()
            n_imfs = np.delete(n_imfs, 7)
        return L._plan.counters(reset=True)[1], n_imfs

    here, ref = spilled(0, False)
    assert here > 0 and spilled(1 << 30, False)[0] == 0
    moved, got = spilled(1 << 30, True)
    assert moved == 0 and np.array_equal(got, ref)
