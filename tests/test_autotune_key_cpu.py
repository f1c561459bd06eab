"""Entries of the autotune cache file hold for the library build that timed
them: another build's, and those of earlier key generations, are not taken."""
import json

import numpy as np
import pytest

from cuda_emd import _native
from cuda_emd import ragged as R


@pytest.fixture
def build(monkeypatch, tmp_path):
    import torch
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d: "B200")
    monkeypatch.setattr(torch.cuda, "get_device_properties",
                        lambda d: type("P", (), {"multi_processor_count": 148}))

    def at(content):
        lib = tmp_path / "lib.so"
        lib.write_bytes(content)
        monkeypatch.setattr(_native, "LIB_PATH", str(lib))
        _native.build_digest.cache_clear()
    yield at
    _native.build_digest.cache_clear()


class _Tier:
    edge, idx = 4096, np.arange(10)

    def __init__(self):
        self.tuning = None
        self.plan = None

    def set_tuning(self, variant, arena):
        self.tuning = (variant, arena)


def _tune(path):
    """The tuning a runner takes without timing anything; None if it has to time."""
    r, t = R.RaggedRunner(device=0, cache_path=path, autotune=False), _Tier()
    chosen = r.tune(None, None, None, [t])
    return t.tuning if chosen else None


def test_entries_hold_for_the_build_that_timed_them(build, tmp_path, monkeypatch):
    monkeypatch.setattr(R, "candidates", lambda plan, n: [(4, 0), (1, 0)])
    path = str(tmp_path / "tune.json")
    build(b"one")
    key = R.RaggedRunner(device=0, cache_path=path)._key(4096)
    old = "t3|B200|" + key.split("|B200|")[1]
    entry = {"variant": 2, "arena": 0, "sample": 10}
    json.dump({old: entry}, open(path, "w"))
    assert _tune(path) is None
    json.dump({old: entry, key: dict(entry, variant=1)}, open(path, "w"))
    assert _tune(path) == (1, 0)
    build(b"two")
    assert _tune(path) is None
    build(b"one")
    assert _tune(path) == (1, 0)
