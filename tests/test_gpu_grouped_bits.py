"""Grouped pairs at the key widths where their sort changes: one sort up to 64 bits,
the bits below the top word sorted first up to 72, ties ordered after the sort past
that -- with long runs of equal top words whose low bits differ.  Against the
oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", (63, 64, 65, 71, 72, 73, 74, 79))
@pytest.mark.parametrize("pairs", (3, 700, 40000))
def test_key_widths_match_oracle(cuda_device, oracle, bits, pairs):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(4096, 11)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    t, ps = yb.build_tree(P, M, leaf_size=4, return_reordered=True)[:2]
    g = yb.compute_tree_geometry(t, ps)
    cpu = lambda x: x.detach().cpu().numpy()  # noqa: E731
    level = cpu(t.node_level)
    one = int(np.bincount(level).argmax())  # all pairs between nodes of one level
    pool = np.flatnonzero(level == one)
    lo, hi = cpu(t.bounds_min), cpu(t.bounds_max)
    cell = (hi - lo).astype(np.float64) / 2.0 ** one
    rng = np.random.default_rng(bits)
    # x and y from a few places (24 bits each at most), z from many
    width = (24, 24, bits - 48)
    centers = np.zeros((level.shape[0], 3))
    for a, w in enumerate(width):
        far = 2.0 ** (w - 1) * 0.6  # differences of up to 1.2 * 2^(w - 1): w bits with sign
        places = rng.uniform(-far / 2, far / 2, 3 if a < 2 else 200)
        places[:2] = -far / 2, far / 2
        centers[:, a] = places[rng.integers(0, places.size, level.shape[0])] * cell[a]
    ends = pool[:2]
    centers[ends[0]], centers[ends[1]] = [[s * 2.0 ** (w - 1) * 0.3 * cell[a] for a, w in
                                           enumerate(width)] for s in (-1, 1)]
    centers = centers.astype(np.float32)
    src, tgt = rng.choice(pool, pairs), rng.choice(pool[:40], pairs)
    src[:2], tgt[:2] = ends, ends[::-1]
    geo = g._replace(center=torch.from_numpy(centers).to(cuda_device))
    got = yb.build_grouped_interactions_from_pairs(
        t, geo, torch.from_numpy(src.astype(np.int64)).to(cuda_device),
        torch.from_numpy(tgt.astype(np.int64)).to(cuda_device))
    want = oracle.grouped_from_pairs(src, tgt, level, centers, lo, hi)
    for k, w in want.items():
        np.testing.assert_array_equal(cpu(getattr(got, k)), w, err_msg=k)
    keys = cpu(got.class_keys).astype(np.int64)
    assert sum(int(x).bit_length() for x in keys.max(0) - keys.min(0)) == bits
