"""The unordered per-target walk at the edges of its two kernels: trees below
2^24 nodes walk sibling pairs with 32-bit candidates, larger trees keep
64-bit ones.  Both must give the lists of the generation-by-generation walk
(schedule "log", itself held to the oracle in test_gpu_parity.py), from the
smallest tree that has pairs to one just past the dispatch line."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


SMALL = [
    (2, 1, 0.6, 128),       # two leaves: one sibling pair
    (3, 1, 0.6, 128),
    (33, 1, 0.6, 1),
    (5000, 1, 0.4, 1),      # every piece hands its rest off
    (20000, 8, 0.3, 3),     # rows past a staging buffer, shared split lists
]
# 16,777,217 nodes: one past the 24-bit slots (one-particle leaves are outside
# what the capacity predictor was trained on, so without its row slots)
LARGE = (8_388_609, 1, 3.0, 128)


@pytest.mark.parametrize("mode,n,leaf,theta,budget",
                         [(m, *c) for m in ("target", "learned") for c in SMALL]
                         + [("target", *LARGE)])
def test_lists_match_log_walk(cuda_device, mode, n, leaf, theta, budget):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs
    from yggdrax_b200 import interactions as I
    from test_gpu_target import _run

    pos, mass = inputs.uniform_cube(n, 5)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tree, ps = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[:2]
    geom = yb.compute_tree_geometry(tree, ps)
    total = int(tree.parent.shape[0])
    assert (total > I._PAIR_WALK_MAX_NODES) == (n > 8_000_000)
    if n > 8_000_000:  # the defaults allow for far longer rows than theta 3 has
        I._TARGET_HINTS[I._hint_key("dehnen", theta, total, mode)] = [24.0] * 8
    yb.set_reference_limits(False)
    yb.set_dense_neighbor_budget(1 << 28)
    try:
        a, an, ares, st = _run(yb, tree, geom, theta, "dehnen", budget, mode)
        assert st["mode"] == mode
        b, bn, bres, st = _run(yb, tree, geom, theta, "dehnen", mode="log")
        assert st["mode"] == "log"
    finally:
        yb.set_reference_limits(True)
        yb.set_dense_neighbor_budget(None)
    for f in ("offsets", "counts", "sources", "targets", "level_offsets", "target_levels"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f
    for f in ("offsets", "counts", "neighbors", "neighbor_leaf_positions"):
        assert torch.equal(getattr(an, f), getattr(bn, f)), f
    for f in ("accept_decisions", "near_decisions", "refine_decisions"):
        assert int(getattr(ares, f)) == int(getattr(bres, f)), f
    assert np.isfinite(float(geom.radius.max()))
