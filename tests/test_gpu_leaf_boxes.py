"""Leaf boxes at the edges of the refit's lane groups (8 lanes per leaf up to
64 particles on average, 32 above): ragged last leaves, leaves of one particle,
a last warp of few leaves, NaN positions -- against the oracle, bit for bit,
and batched against single trees."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(2, 1), (31, 1), (33, 1), (257, 8), (264, 8), (4129, 32),
                                    (4160, 63), (6464, 64), (6500, 65), (5000, 200), (999, 1000)])
@pytest.mark.parametrize("nan", (False, True))
def test_leaf_boxes_match_oracle(cuda_device, oracle, n, leaf, nan):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.plummer(n, n)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tree, ps = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[:2]
    ot = oracle.build_tree(pos, mass, leaf_size=leaf)
    want_ps = ot.positions_sorted.copy()
    if nan:
        ps = ps.clone()
        ps[n // 2, 1] = float("nan")
        want_ps[n // 2, 1] = np.nan
    got = yb.compute_tree_geometry(tree, ps)
    want = oracle.compute_tree_geometry(ot, want_ps)
    for f in ("center", "half_extent", "radius", "max_extent"):
        np.testing.assert_array_equal(getattr(got, f).cpu().numpy(), getattr(want, f), err_msg=f)


@pytest.mark.parametrize("leaf", (1, 16, 64, 65))
def test_batched_leaf_boxes(cuda_device, leaf):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import batch, inputs

    sizes = [1, 2, 63, 64, 65, 700, 4097]
    off = np.concatenate([[0], np.cumsum(sizes)])
    pos, mass = inputs.plummer(int(off[-1]), 4)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    bt = batch.build_trees_batched(P, M, torch.from_numpy(off), leaf_size=leaf)
    bg = batch.compute_tree_geometry_batched(bt)
    for i, (a, b) in enumerate(zip(off[:-1], off[1:])):
        t, ps = yb.build_tree(P[a:b].contiguous(), M[a:b].contiguous(), leaf_size=leaf,
                              return_reordered=True)[:2]
        g = yb.compute_tree_geometry(t, ps)
        for x, y in zip(bg.geometry(bt, i), g):
            assert torch.equal(x, y), i
