"""The ragged runner's cached plan follows the lengths of the batch it is given,
whatever buffers they come in: the same buffers refilled, the same offsets in
other buffers, with the offsets read from the tensor and given by the host."""
import numpy as np
import pytest
import torch

from cuda_emd import ragged as R


class _Tier:
    """A tier without its device plan."""

    def __init__(self, edge, idx, cfg, device):
        self.edge, self.idx, self.max_n, self.variant, self.arena = edge, idx, 0, 4, 0


@pytest.fixture
def runner(monkeypatch):
    monkeypatch.setattr(R, "Tier", _Tier)
    monkeypatch.setattr(R.RaggedRunner, "tune", lambda self, *a, **k: {})
    return R.RaggedRunner(device=0, cache_path=None)


def _offsets(lens):
    return np.r_[0, np.cumsum(lens)].astype(np.int64)


def _plan(r, values, offsets, host):
    tiers, orders = r.prepare(values, offsets, offsets_host=offsets.numpy().copy() if host else None)
    return {t.edge: o.tolist() for t, o in zip(tiers, orders)}


@pytest.mark.parametrize("host", [False, True])
def test_refilled_buffers_are_planned_again(runner, host):
    values = torch.zeros(6000, dtype=torch.float64)
    offsets = torch.from_numpy(_offsets([500, 3000, 600, 1900]))
    assert _plan(runner, values, offsets, host) == {4096: [1], 2048: [3], 1024: [0, 2]}
    first = runner._prep
    assert _plan(runner, values, offsets, host) == {4096: [1], 2048: [3], 1024: [0, 2]}
    assert runner._prep is first                      # the same lengths: the same plan
    offsets.numpy()[:] = _offsets([3000, 500, 1900, 600])     # not through torch: no version change
    assert _plan(runner, values, offsets, host) == {4096: [0], 2048: [2], 1024: [1, 3]}


@pytest.mark.parametrize("host", [False, True])
def test_equal_lengths_in_other_buffers_share_the_plan(runner, host):
    lens = [100, 1500, 700]
    a = _plan(runner, torch.zeros(2300, dtype=torch.float64), torch.from_numpy(_offsets(lens)), host)
    first = runner._prep
    assert _plan(runner, torch.ones(2300, dtype=torch.float64), torch.from_numpy(_offsets(lens)), host) == a
    assert runner._prep is first
    with torch.inference_mode():
        offsets = torch.from_numpy(_offsets(lens)).clone()
        assert _plan(runner, torch.ones(2300, dtype=torch.float64), offsets, host) == a


def test_offsets_given_as_a_reused_host_array(runner):
    values, off_h = torch.zeros(6000, dtype=torch.float64), _offsets([500, 3000])
    offsets = torch.from_numpy(off_h)
    assert [t.edge for t in runner.prepare(values, offsets, offsets_host=off_h)[0]] == [4096, 1024]
    off_h[1] = 3000
    off_h[2] = 3000 + 3000
    assert [t.edge for t in runner.prepare(values, offsets, offsets_host=off_h)[0]] == [4096]
