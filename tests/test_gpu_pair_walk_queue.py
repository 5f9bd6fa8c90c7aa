"""A pair walk whose queue is too short ends at once: a warp goes on with a target's
left child only if its last push of a right child found room.  So a chain of k
left children has queued k - 1, and with at most one chain per queue slot at most
three targets run per slot.  (Going on regardless ran whole chains.)"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("queue", (2, 3, 64, 1000))
def test_pieces_are_bounded_by_the_queue(cuda_device, queue):
    import torch

    from yggdrax_b200 import _lib as L
    from yggdrax_b200 import batch as B

    lib, n = L.lib(), 40000
    pos = torch.rand(n, 3, generator=torch.Generator().manual_seed(4)).to(cuda_device)
    bt = B.build_trees_batched(pos, torch.ones_like(pos[:, 0]), [0, n], leaf_size=4)
    bg = B.compute_tree_geometry_batched(bt)
    total, leaves = bt.total_nodes, bt.total_leaves
    caps = np.asarray([1 << 23] * 4 + [1 << 18] * 3 + [queue], np.int64)
    ws = L.workspace(lib.ygx_batch_target_walk_workspace_size(total, leaves, caps.ctypes.data),
                     cuda_device)
    stats, needs = np.zeros(L.TSTAT_WORDS, np.uint64), np.zeros(14, np.uint64)
    flags = np.zeros(1, np.uint32)
    rc = lib.ygx_batch_target_walk(
        L.ptr(bg.center), L.ptr(bg.radius), L.ptr(bg.max_extent), L.ptr(bt.left32),
        L.ptr(bt.right32), L.ptr(bt.leafpos32), L.ptr(bt.level32), total, leaves,
        L.ptr(bt.leaf_off), 1, L.ptr(bt.seg_flags), 0, 0.5, 1.0, caps.ctypes.data,
        stats.ctypes.data, needs.ctypes.data, flags.ctypes.data, L.ptr(ws), ws.numel(),
        L.stream_handle(cuda_device))
    assert rc == 0 and int(flags[0]) == L.FLAG_LOG_OVERFLOW
    assert int(needs[7]) > queue  # asks for more room
    assert 0 < int(needs[11]) <= 3 * queue
