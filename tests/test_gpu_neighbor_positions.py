"""The dense neighbour position table at the edges of its split (a warp per
128 columns of a row): equal to the table built from the lists by torch."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,theta", [
    (16, 8, 0.01),       # one neighbour
    (129 * 8, 8, 0.01),  # 128 columns: one full part
    (130 * 8, 8, 0.01),  # 129: a second part of one column
    (257 * 8, 8, 0.01),  # 256
    (30000, 8, 0.4),     # rows much shorter than the longest
])
def test_positions_match_lists(cuda_device, n, leaf, theta):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(n, 11)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tree, ps = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[:2]
    geom = yb.compute_tree_geometry(tree, ps)
    yb.set_reference_limits(False)
    yb.set_dense_neighbor_budget(1 << 28)
    try:
        _, near = yb.build_interactions_and_neighbors(tree, geom, theta=theta, mac_type="bh")
    finally:
        yb.set_reference_limits(True)
        yb.set_dense_neighbor_budget(None)
    rows, width = near.neighbor_leaf_positions.shape
    if theta < 0.1:
        assert width == rows - 1
    assert width == int(near.counts.max())
    pos_of = torch.full((int(tree.parent.shape[0]),), -1, dtype=torch.int64, device=cuda_device)
    pos_of[near.leaf_indices.long()] = torch.arange(rows, device=cuda_device)
    want = torch.full((rows, width), -1, dtype=torch.int64, device=cuda_device)
    row = torch.repeat_interleave(torch.arange(rows, device=cuda_device), near.counts.long())
    col = torch.arange(row.numel(), device=cuda_device) - near.offsets.long()[row]
    want[row, col] = pos_of[near.neighbors.long()]
    assert torch.equal(near.neighbor_leaf_positions.long(), want)
