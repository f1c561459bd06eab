"""warmup() launches the kernel instances of small and of large batches, allocates
their scratch, and leaves the plan as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", ["double", "float"])
@pytest.mark.parametrize("n", [64, 3000])
def test_warmup_allocates_the_scratch_and_keeps_the_plan(real, n):
    import torch
    from cuda_emd import EMDKernelConfig, GPUBatchEMD, workloads as W
    cfg = EMDKernelConfig(real_t=real)
    X = torch.from_numpy(W.sinusoid_batch(900, n, seed=1).astype(cfg.dtype)).cuda()
    first = GPUBatchEMD(cfg)                     # loads the modules
    first.warmup(n)
    plan = EMDKernelConfig(real_t=real).build()._plan
    ctas = plan.query(n, first.config.f32)[1]
    assert ctas == (4 if real == "float" else 2) if n == 3000 else ctas == (5 if real == "float" else 4)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for batch, x in ((None, X[:sms]), (900, X), (900, X[:sms]), (900, X[:500])):
        first(x)                                 # fills torch's cache of outputs
        emd = GPUBatchEMD(cfg)
        emd.warmup(n, batch)
        torch.cuda.synchronize()
        assert tuple(emd.last_debug[0].shape) == (1, cfg.max_imfs)
        free = torch.cuda.mem_get_info()[0]
        emd(x)
        torch.cuda.synchronize()
        assert free - torch.cuda.mem_get_info()[0] < 4 << 20, batch
    assert emd._launcher._plan.by_length()
    for a, b in zip(first(X), emd(X)):
        assert torch.equal(a, b)


def test_warmup_keeps_an_instance_that_was_set():
    import torch
    from cuda_emd import GPUBatchEMD
    emd = GPUBatchEMD()
    plan = emd._get_launcher()._plan
    plan.set_variant(2)
    emd.warmup()
    assert plan._variant == 2
    plan.set_variant(0)
    plan.set_arena(60000)
    emd.warmup()
    assert (plan._variant, plan._arena) == (0, 60000)
