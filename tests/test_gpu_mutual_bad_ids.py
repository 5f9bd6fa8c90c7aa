"""The mutual walk reports a child id outside the tree also where later pairs of
the same thread hold a missing child (-1), which by itself is passed over."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", (False, True))
def test_child_outside_the_tree_is_reported(cuda_device, bad):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import _lib as L

    depth = 16  # a complete tree; the last internal level has no right children
    ni = 2 ** depth - 1
    total = 2 * ni + 1
    i = torch.arange(ni, dtype=torch.int64, device=cuda_device)
    left = torch.full((total,), -1, dtype=torch.int64, device=cuda_device)
    right = left.clone()
    left[:ni], right[:ni] = 2 * i + 1, 2 * i + 2
    first = 2 ** (depth - 1) - 1
    right[first:ni] = -1
    # all nodes on one spot, so every pair is refined, but one node far away:
    # only its pair with itself is, 16 generations down among half a million
    odd = first + 3
    right[odd] = 2 * odd + 2
    if bad:
        left[odd] = total + 7
    centers = torch.zeros((total, 3), device=cuda_device)
    centers[odd] = 1e6
    radii = torch.ones(total, device=cuda_device)
    run = lambda: yb.dual_tree_walk_mutual(left, right, centers, radii, 0.5, 0,  # noqa: E731
                                           max_pair_queue=1 << 22, far_cap=1 << 22,
                                           near_cap=1 << 22)
    if bad:
        with pytest.raises(L.YgxError, match="YGX_ERR_ARG"):
            run()
    else:
        assert int(run().far_count) > 0
