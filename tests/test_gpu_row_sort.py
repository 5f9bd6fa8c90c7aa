"""The row finalize: rows of every size class, sorted by warps, by groups of
warps and through the bitmap, equal the lists whose rows the walk itself
orders (schedule "target_ordered", no row sort)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# upper ends of the size classes
CLASSES = [32, 64, 96, 128, 192, 256, 384, 512, 768, 1024, 1536, 2048, 3072, 4096, 6144, 8192,
           16384, 65536]


@pytest.mark.parametrize("points,n,leaf,theta", [
    ("uniform_cube", 30, 8, 0.5),        # a few short rows, no long ones
    ("uniform_cube", 30000, 4, 0.3),
    ("uniform_cube", 100000, 8, 0.25),   # several rows of every group size
    ("plummer", 300000, 4, 0.45),        # halo leaves with very long rows
])
def test_rows_equal_ordered_walk(cuda_device, points, n, leaf, theta):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs
    from test_gpu_target import _run

    pos, mass = getattr(inputs, points)(n, 3)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tree, ps = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[:2]
    geom = yb.compute_tree_geometry(tree, ps)
    yb.set_reference_limits(False)
    yb.set_dense_neighbor_budget(1 << 28)
    try:
        want, want_n, _, st = _run(yb, tree, geom, theta, "bh", mode="target_ordered")
        assert st["mode"] == "target_ordered"
        for mode in ("target", "learned"):
            got, got_n, _, st = _run(yb, tree, geom, theta, "bh", mode=mode)
            assert st["mode"] == mode
            for f in ("offsets", "counts", "sources", "targets", "target_levels"):
                assert torch.equal(getattr(got, f), getattr(want, f)), (mode, f)
            for f in ("offsets", "counts", "neighbors"):
                assert torch.equal(getattr(got_n, f), getattr(want_n, f)), (mode, f)
    finally:
        yb.set_reference_limits(True)
        yb.set_dense_neighbor_budget(None)
    counts = np.concatenate([want.counts.cpu().numpy(), want_n.counts.cpu().numpy()])
    seen = set(np.searchsorted(CLASSES, counts[counts > 0]).tolist())
    if n == 100000:
        assert seen >= set(range(16))
    if points == "plummer":
        assert max(seen) >= 17
