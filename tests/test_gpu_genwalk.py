"""The mutual and native octree walks at the sizes where their one-launch
compaction can go wrong: wavefronts below one chunk (512 pairs), of many chunks
per CTA, children of eight-way cells, both index dtypes' capacities met
exactly, and a grid barrier that gives up (an error code, no fault)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,theta", [(2, 1, 0.6), (9, 1, 0.9), (700, 4, 0.6),
                                          (30000, 2, 0.35)])
def test_mutual_walk_sizes(cuda_device, oracle, n, leaf, theta):
    import torch

    import yggdrax_b200 as yb
    from test_gpu_mutual import FIELDS, _check
    from yggdrax_b200 import inputs

    pos, mass = inputs.plummer(n, 21)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tr, ps = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[:2]
    g = yb.compute_tree_geometry(tr, ps)
    total, ni = int(tr.parent.shape[0]), int(tr.left_child.shape[0])
    lf = torch.full((total,), -1, dtype=torch.int64, device=cuda_device)
    rt = lf.clone()
    lf[:ni], rt[:ni] = tr.left_child, tr.right_child
    host = [x.cpu().numpy() for x in (lf, rt, g.center, g.radius)]
    big = dict(max_pair_queue=1 << 23, far_cap=1 << 23, near_cap=1 << 23)
    want = oracle.dual_tree_walk_mutual(*host, theta, 0, **big)
    far, near = max(1, int(want["far_count"])), max(1, int(want["near_count"]))
    for caps in (big, dict(max_pair_queue=1 << 23, far_cap=far, near_cap=near),
                 dict(max_pair_queue=1 << 23, far_cap=max(1, far - 1), near_cap=near)):
        want = oracle.dual_tree_walk_mutual(*host, theta, 0, **caps)
        got = yb.dual_tree_walk_mutual(lf, rt, g.center, g.radius, theta, 0, **caps)
        _check(got, want, (n, leaf, theta, caps))
    assert len(FIELDS) == 9


@pytest.mark.parametrize("n,depth,theta", [(9, 1, 0.6), (600, 2, 0.9), (200000, 5, 0.6)])
def test_octree_walk_sizes(cuda_device, oracle, n, depth, theta):
    import torch

    import yggdrax_b200 as yb
    from test_gpu_octwalk import NEAR_FIELDS, OCT_FIELDS, _np
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(n, 9)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    topo = yb.build_fixed_depth_octree(P, M, target_leaf_particles=2, max_depth=depth,
                                       return_reordered=True)[0].topology
    fields = {k: _np(getattr(topo, k)) for k in OCT_FIELDS}
    v = oracle.octree_traversal_view(fields, int(topo.left_child.shape[0]),
                                     _np(topo.bounds_min), _np(topo.bounds_max))
    kw = dict(max_interactions_per_node=1 << 20, max_neighbors_per_leaf=1 << 20,
              max_pair_queue=1 << 24)
    cfg = yb.DualTreeTraversalConfig(process_block=64, **kw)
    far = oracle.octree_native_walk(v, theta, "dehnen", collect_far=True, collect_near=False, **kw)
    near = oracle.octree_native_walk(v, theta, "dehnen", collect_far=False, collect_near=True,
                                     **kw)
    fp = yb.build_octree_native_far_pairs(topo, None, theta=theta, mac_type="dehnen",
                                          traversal_config=cfg)
    assert np.array_equal(_np(fp.targets), far["targets"])
    assert np.array_equal(_np(fp.sources), far["sources"])
    nb = yb.build_octree_native_neighbor_lists(topo, None, theta=theta, mac_type="dehnen",
                                               traversal_config=cfg)
    nl = oracle.octree_native_neighbor_list(near, fields["oct_node_ranges"])
    for f in NEAR_FIELDS + ("neighbors", "neighbor_leaf_positions"):
        assert np.array_equal(_np(getattr(nb, f)), nl[f]), f


def test_barrier_limit_is_an_error_not_a_hang(cuda_device):
    """With no polls allowed the grid barrier gives up at once: the call
    returns an error, and the next call at the default limit is right."""
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import _lib as L
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(20000, 2)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    tr, ps = yb.build_tree(P, M, leaf_size=8, return_reordered=True)[:2]
    g = yb.compute_tree_geometry(tr, ps)
    total, ni = int(tr.parent.shape[0]), int(tr.left_child.shape[0])
    lf = torch.full((total,), -1, dtype=torch.int64, device=cuda_device)
    rt = lf.clone()
    lf[:ni], rt[:ni] = tr.left_child, tr.right_child
    run = lambda: yb.dual_tree_walk_mutual(lf, rt, g.center, g.radius, 0.6, 0,  # noqa: E731
                                           max_pair_queue=1 << 22, far_cap=1 << 22,
                                           near_cap=1 << 22)
    want = run()
    lib = L.lib()
    old = np.zeros(1, np.int32)
    L.check(lib.ygx_tune_get(L.TUNE["spin_limit"], old.ctypes.data), "ygx_tune_get")
    L.check(lib.ygx_tune_set(L.TUNE["spin_limit"], 0), "ygx_tune_set")
    try:
        with pytest.raises(L.YgxError, match="YGX_ERR_TIMEOUT"):
            run()
    finally:
        L.check(lib.ygx_tune_set(L.TUNE["spin_limit"], int(old[0])), "ygx_tune_set")
    got = run()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
