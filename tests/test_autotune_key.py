"""What a cached tuning choice is kept for."""
from types import SimpleNamespace

import numpy as np

from kiddo_b200 import autotune


def _builder(nq, n=1_000_000, k=8):
    tree = SimpleNamespace(dtype=np.float32, dims=3, size=lambda: n)
    return SimpleNamespace(tree=tree, family=2, metric=0, max_qty=k, box=None,
                           queries=np.empty((nq, 3), np.float32))


def test_a_choice_holds_for_batches_of_its_size():
    """A small batch takes another engine than a large one."""
    assert autotune.key_for(_builder(64)) != autotune.key_for(_builder(1 << 20))
    assert autotune.key_for(_builder(1 << 20)) == autotune.key_for(_builder((1 << 21) + 5))
    assert autotune.key_for(_builder(1 << 20)) != autotune.key_for(_builder(1 << 22))
    assert autotune.key_for(_builder(0)) == autotune.key_for(_builder(1))


def test_a_choice_tuned_on_a_large_batch_is_not_found_for_a_small_one(tmp_path, monkeypatch):
    monkeypatch.setenv("KIDDO_B200_TUNE_CACHE", str(tmp_path / "tune.json"))
    large = _builder(1 << 20)
    autotune._store({autotune.key_for(large): {"engine": "thread", "spatial_order": True}})
    assert autotune.lookup(large)["engine"] == "thread"
    assert autotune.lookup(_builder(64)) is None
