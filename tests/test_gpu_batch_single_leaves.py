"""Batches whose sets are single leaves: trees of one node, no pairs."""
import numpy as np
import pytest
import torch

from yggdrax_b200 import batch as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sets,points,leaf", [(1, 1, 1), (3, 5, 8), (60000, 5, 8)])
def test_sets_of_one_leaf(cuda_device, sets, points, leaf):
    off = np.arange(sets + 1, dtype=np.int64) * points
    pos = torch.rand(int(off[-1]), 3, generator=torch.Generator().manual_seed(1)).to(cuda_device)
    bt = B.build_trees_batched(pos, torch.ones_like(pos[:, 0]), off, leaf_size=leaf)
    bg = B.compute_tree_geometry_batched(bt)
    bi = B.build_interactions_and_neighbors_batched(bt, bg, theta=0.5, mac_type="bh")
    assert bt.total_nodes == sets and bi.sources.numel() == 0 and bi.neighbors.numel() == 0
    assert bool((bt.parent == -1).all()) and bool((bt.num_levels == 1).all())
    p = bt.positions_sorted.view(sets, points, 3)
    lo, hi = p.amin(1), p.amax(1)
    assert torch.equal(bg.center, 0.5 * (lo + hi))
    assert not bool(bt.seg_flags.any())
    assert torch.equal(bt.nodes_by_level, torch.zeros_like(bt.nodes_by_level))
