"""The lists' plan (several scans in one go) at the edges of its tiles: trees
whose node or leaf counts sit at a tile (4096), at the largest size that runs
in one launch (65,536 values) and past it; every table against the log
schedule's."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ("learned", "target", "target_ordered"))
@pytest.mark.parametrize("leaves", (2, 2048, 2049, 4096, 32768, 32769, 65537))
def test_tables_at_tile_edges(cuda_device, mode, leaves):
    import torch

    import yggdrax_b200 as yb
    from test_gpu_target import _run
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(2 * leaves, leaves)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tree, ps = yb.build_tree(P, M, leaf_size=2, return_reordered=True)[:2]
    assert int(tree.parent.shape[0]) == 2 * leaves - 1
    geom = yb.compute_tree_geometry(tree, ps)
    yb.set_reference_limits(False)
    yb.set_dense_neighbor_budget(1 << 28)
    try:
        a, an, _, st = _run(yb, tree, geom, 0.9, "dehnen", mode=mode)
        assert st["mode"] == mode
        b, bn, _, _ = _run(yb, tree, geom, 0.9, "dehnen", mode="log")
    finally:
        yb.set_reference_limits(True)
        yb.set_dense_neighbor_budget(None)
    for f in ("offsets", "counts", "sources", "targets", "level_offsets", "target_levels"):
        assert torch.equal(getattr(a, f), getattr(b, f)), f
    for f in ("offsets", "counts", "neighbors", "neighbor_leaf_positions"):
        assert torch.equal(getattr(an, f), getattr(bn, f)), f
