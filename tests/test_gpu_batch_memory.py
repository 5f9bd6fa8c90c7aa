"""Batched lists where the per-target walk's pools do not fit the memory: the
generation walk's come instead."""
import numpy as np
import pytest
import torch

from yggdrax_b200 import _lib as L
from yggdrax_b200 import batch as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("failing", (1, 2))
def test_out_of_memory_takes_the_generation_walk(cuda_device, monkeypatch, failing):
    off = np.arange(11, dtype=np.int64) * 900
    pos = torch.rand(int(off[-1]), 3, generator=torch.Generator().manual_seed(2)).to(cuda_device)
    bt = B.build_trees_batched(pos, torch.ones_like(pos[:, 0]), off, leaf_size=8)
    bg = B.compute_tree_geometry_batched(bt)
    want = B._log_lists_batched(bt, bg, 0.5, "bh", 1.0)
    real, state = B._target_lists_batched, dict(calls=0)

    def target(*args):
        def workspace(nbytes, dev, zero=True):
            state["calls"] += 1
            if state["calls"] >= failing:  # the first pools, or those of a re-run
                raise torch.cuda.OutOfMemoryError("no room")
            return plain(nbytes, dev, zero)

        plain = L.workspace
        with monkeypatch.context() as m:
            m.setattr(L, "workspace", workspace)
            if failing == 2:
                m.setattr(B, "_BATCH_FIRST_CAPS", [1e-6] * 8)
                m.setattr(B, "_target_caps", lambda total, nl, hint: [64] * 8)
            return real(*args)

    monkeypatch.setattr(B, "_target_lists_batched", target)
    got = B.build_interactions_and_neighbors_batched(bt, bg, theta=0.5, mac_type="bh")
    assert state["calls"] == failing
    for name in ("node_offsets", "far_counts", "sources", "targets", "target_levels",
                 "near_offsets", "near_counts", "neighbors"):
        assert torch.equal(getattr(got, name), getattr(want, name)), name
