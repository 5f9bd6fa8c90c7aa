"""Batched lists by the per-target walk over the forest, against the
generation walk on the same trees: every table equal, integer for integer."""
import numpy as np
import pytest
import torch

from yggdrax_b200 import batch as B
from yggdrax_b200 import interactions as I

pytestmark = pytest.mark.gpu

TABLES = ("node_offsets", "far_counts", "sources", "targets", "target_levels",
          "near_offsets", "near_counts", "neighbors")
STATS = ("far_total", "near_total", "max_far", "max_near", "accept", "near", "refine")


def _sets(sizes, seed=5, clump=False):
    g = torch.Generator().manual_seed(seed)
    n = int(sum(sizes))
    pos = torch.rand(n, 3, generator=g)
    if clump:
        pos = pos ** 6
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    return pos.cuda(), torch.ones(n).cuda(), off


@pytest.mark.parametrize("mac,theta", [("bh", 0.5), ("dehnen", 0.6), ("engblom", 0.4)])
@pytest.mark.parametrize("sizes,leaf,clump", [
    ([9], 4, False),                      # one set, its root's children leaves
    ([1, 2, 1, 3, 200, 1], 2, False),     # sets of one leaf beside larger ones
    ([5, 900, 33, 4000, 64], 8, True),    # ragged
    ([130] * 700, 4, False),              # more sets than CTAs
    ([30000, 2], 16, False),
])
def test_equal_to_generation_walk(sizes, leaf, clump, mac, theta):
    pos, mass, off = _sets(sizes, clump=clump)
    bt = B.build_trees_batched(pos, mass, off, leaf_size=leaf)
    bg = B.compute_tree_geometry_batched(bt)
    want = B._log_lists_batched(bt, bg, theta, mac, 1.25)
    for hints in (False, True):  # default capacities, then the learned ones
        if not hints:
            I._TARGET_HINTS.clear()
        got = B._target_lists_batched(bt, bg, theta, mac, 1.25)
        for name in TABLES:
            assert torch.equal(getattr(got, name), getattr(want, name)), name
        assert {k: got.stats[k] for k in STATS} == {k: want.stats[k] for k in STATS}


def test_overflow_reruns():
    """Capacities far too small for the forest are grown to fit."""
    pos, mass, off = _sets([3000] * 40)
    bt = B.build_trees_batched(pos, mass, off, leaf_size=4)
    bg = B.compute_tree_geometry_batched(bt)
    want = B._log_lists_batched(bt, bg, 0.3, "bh", 1.0)
    I._TARGET_HINTS.clear()
    I._TARGET_HINTS[B._hint_key("bh", 0.3, bt.total_nodes, "batch_target")] = [1e-6] * 8
    got = B._target_lists_batched(bt, bg, 0.3, "bh", 1.0)
    for name in TABLES:
        assert torch.equal(getattr(got, name), getattr(want, name)), name


def test_tied_codes_take_the_generation_walk():
    pos, mass, off = _sets([64, 300])
    pos[:64] = pos[:1].clone()  # every code of the first set equal
    bt = B.build_trees_batched(pos, mass, off, leaf_size=4)
    bg = B.compute_tree_geometry_batched(bt)
    assert bool((bt.seg_flags != 0).any())
    assert B._target_lists_batched(bt, bg, 0.5, "bh", 1.0) is None
    want = B._log_lists_batched(bt, bg, 0.5, "bh", 1.0)
    got = B.build_interactions_and_neighbors_batched(bt, bg, theta=0.5, mac_type="bh")
    for name in TABLES:
        assert torch.equal(getattr(got, name), getattr(want, name)), name


def test_extents_refused():
    pos, mass, off = _sets([100, 100])
    bt = B.build_trees_batched(pos, mass, off, leaf_size=8)
    bg = B.compute_tree_geometry_batched(bt)
    bg.max_extent[3] = 0.0
    with pytest.raises(ValueError, match="extents must be positive"):
        B.build_interactions_and_neighbors_batched(bt, bg, theta=0.5, mac_type="bh")
