"""The default schedule past 2^24 nodes: predicted row slots on the walk with
64-bit candidates (smaller trees take the walk over sibling pairs), rows written
in place and rows that outgrew their slots, against the generation walk."""

import pytest

pytestmark = pytest.mark.gpu


def test_predicted_rows_past_the_slots_range(cuda_device):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs
    from yggdrax_b200 import interactions as I
    from test_gpu_target import _run

    theta = 3.0  # short rows: 24 M entries in all
    pos, mass = inputs.uniform_cube(16_777_231, 5)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tree, ps = yb.build_tree(P, M, leaf_size=2, return_reordered=True)[:2]
    geom = yb.compute_tree_geometry(tree, ps)
    total = int(tree.parent.shape[0])
    assert total > I._PAIR_WALK_MAX_NODES
    # (the defaults allow for far longer rows)
    I._TARGET_HINTS[I._hint_key("dehnen", theta, total, "learned")] = [24.0] * 8
    yb.set_reference_limits(False)
    yb.set_dense_neighbor_budget(1 << 28)
    try:
        a, an, ares, st = _run(yb, tree, geom, theta, "dehnen", None, "learned")
        assert st["mode"] == "learned" and st["padded_far"] > 0
        assert st["ovf_rows"] > 0 and st["ovf_entries"] < st["far_total"] + st["near_total"]
        b, bn, bres, st = _run(yb, tree, geom, theta, "dehnen", mode="log")
        assert st["mode"] == "log"
    finally:
        yb.set_reference_limits(True)
        yb.set_dense_neighbor_budget(None)
    for f in ("offsets", "counts", "sources", "targets", "level_offsets", "target_levels"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f
    for f in ("offsets", "counts", "neighbors"):
        assert torch.equal(getattr(an, f), getattr(bn, f)), f
    for f in ("accept_decisions", "near_decisions", "refine_decisions"):
        assert int(getattr(ares, f)) == int(getattr(bres, f)), f
