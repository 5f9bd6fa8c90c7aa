"""Grouped pairs whose keys tie in their top 64 bits: short runs (ordered in
place), runs of exactly the longest length that is, one longer and far longer
(the list is sorted by the low word first), and pair counts at the tiles' edges
-- every output against the oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tree(cuda_device):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.plummer(60000, 11)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    t, ps = yb.build_tree(P, M, leaf_size=8, return_reordered=True)[:2]
    g = yb.compute_tree_geometry(t, ps)
    far = yb.build_interactions_and_neighbors(t, g, theta=0.6, mac_type="dehnen")[0]
    return t, g, far.sources.cpu().numpy(), far.targets.cpu().numpy()


@pytest.mark.parametrize("pairs,copies", [(1, 0), (2, 0), (4095, 0), (4096, 0), (4097, 0),
                                          (None, 0), (20000, 2), (20000, 1024), (20000, 1025),
                                          (20000, 9000)])
def test_grouped_matches_oracle(cuda_device, oracle, tree, pairs, copies):
    import torch

    import yggdrax_b200 as yb

    t, g, src, tgt = tree
    rng = np.random.default_rng(5)
    if pairs is not None:
        pick = np.sort(rng.choice(src.shape[0], pairs, replace=False))
        src, tgt = src[pick], tgt[pick]
    if copies:  # one pair `copies` times in all, spread over the list
        at = np.sort(rng.integers(0, src.shape[0], copies - 1))
        src, tgt = np.insert(src, at, src[7]), np.insert(tgt, at, tgt[7])
    got = yb.build_grouped_interactions_from_pairs(
        t, g, torch.from_numpy(src).to(cuda_device), torch.from_numpy(tgt).to(cuda_device))
    cpu = lambda x: x.detach().cpu().numpy()  # noqa: E731
    want = oracle.grouped_from_pairs(src, tgt, cpu(t.node_level), cpu(g.center),
                                     cpu(t.bounds_min), cpu(t.bounds_max))
    for k, w in want.items():
        np.testing.assert_array_equal(cpu(getattr(got, k)), w, err_msg=k)
    if pairs is None:  # more than 64 bits: the ties are what is tested here
        span = cpu(got.class_keys).max(0).astype(np.int64) - cpu(got.class_keys).min(0)
        assert sum(int(x).bit_length() for x in span) > 64
