"""ygx_octree_walk's far counts are by cell, whatever row keys the caller gave
the cells: a permutation of the level order here, and keys that are no row at
all (a cell that the caller's level order misses), which only the log carries."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("keys", ("level", "permuted", "outside"))
def test_far_counts_by_cell(cuda_device, keys):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import _lib as L
    from yggdrax_b200 import inputs
    from yggdrax_b200.dtypes import INDEX_BITS, INDEX_DTYPE
    from yggdrax_b200.octree_walk import build_explicit_octree_traversal_view

    dev = cuda_device
    pos, mass = inputs.plummer_clumps(3000, 7)
    P, M_ = torch.from_numpy(pos).to(dev), torch.from_numpy(mass).to(dev)
    tree = yb.build_fixed_depth_octree(P, M_, max_depth=4, return_reordered=True)[0]
    view = build_explicit_octree_traversal_view(getattr(tree, "topology", tree))
    M = int(view.parent.shape[0])
    root = int(torch.argmin(view.parent).item())
    g = torch.Generator(device=dev).manual_seed(1)
    key_of = torch.arange(M, device=dev) if keys == "level" else \
        torch.randperm(M, generator=g, device=dev)
    if keys == "outside":
        key_of[::2] = 2 ** 31 - 1 - key_of[::2]
        key_of[1::4] = -1
    key_of = key_of.to(torch.int32).contiguous()
    children = view.children.to(INDEX_DTYPE).contiguous()
    counts = view.child_counts.to(INDEX_DTYPE).contiguous()
    leaf = view.leaf_mask.to(torch.uint8).contiguous()
    lib, wf, log = L.lib(), 1 << 18, 1 << 20
    key = torch.zeros(log, dtype=torch.int64, device=dev)
    val = torch.zeros(log, dtype=torch.int32, device=dev)
    cnt = torch.zeros(M, dtype=torch.int32, device=dev)
    ws = L.workspace(lib.ygx_octree_walk_workspace_size(M, wf), dev)
    stats, flags = np.zeros(8, np.int64), np.zeros(1, np.uint32)
    rc = lib.ygx_octree_walk(
        L.ptr(children), L.ptr(counts), INDEX_BITS, M, L.ptr(view.box_centers),
        L.ptr(view.box_radii), L.ptr(view.box_max_extents), L.ptr(leaf), L.ptr(key_of), None, M,
        root, 1, 0.6, 1.0, wf, wf, 1 << 20, 1 << 20, log, L.ptr(key), L.ptr(val), None, None,
        L.ptr(cnt), None, stats.ctypes.data, flags.ctypes.data, L.ptr(ws), ws.numel(),
        L.stream_handle(dev))
    assert rc == 0 and int(flags[0]) == 0
    n = int(stats[0])
    assert n > 1000
    # every logged entry names one cell of a pair, and its key the other: the
    # pairs come twice, so a cell stands in as many entries as its row holds
    want = torch.bincount(val[:n].long(), minlength=M).to(torch.int32)
    assert torch.equal(cnt, want)
    have = torch.bincount((key[:n] & 0xffffffff) % 1000003, minlength=1000003)
    rows = torch.zeros_like(have).index_add_(0, (key_of.long() & 0xffffffff) % 1000003, want.long())
    assert torch.equal(have, rows)
