"""Grouped pairs with long runs of equal top words: of one class, of classes in
order, of classes in any order, at the lengths where a warp's ranking, a CTA's sort
and the sort of the whole list take over, and several digits of the rest of the
key.  Centres are made so that target level, source level and the x and y
displacements agree and only z differs.  Every output against the oracle."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RUNS = (2, 31, 32, 33, 255, 256, 257, 511, 512, 513, 1024, 1025, 5000)


@pytest.fixture(scope="module")
def tree(cuda_device):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.plummer(60000, 11)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    t, ps = yb.build_tree(P, M, leaf_size=4, return_reordered=True)[:2]
    return t, yb.compute_tree_geometry(t, ps)


def _pairs(t, lengths, order, rng):
    """(centres, sources, targets): a run of pairs per length."""
    level = t.node_level.cpu().numpy()
    lo, hi = t.bounds_min.cpu().numpy(), t.bounds_max.cpu().numpy()
    centers = np.zeros((level.shape[0], 3), np.float32)
    centers[:] = (lo + hi) / 2
    deep, shallow = int(level.max()), int(np.bincount(level).argmax())
    pool = np.flatnonzero(level == shallow)
    src, tgt = [], []
    cell = ((hi - lo).astype(np.float64) / 2.0 ** shallow).astype(np.float32)
    need = sum(min(n, 40) for n in lengths) + len(lengths)
    assert pool.size > need
    at = 0
    for r, n in enumerate(lengths):
        target, sources = pool[at], pool[at + 1:at + 1 + min(n, 40)]
        at += 1 + sources.size
        # (a displacement in x of its own per run; z spread over many cells)
        centers[target] = lo
        centers[sources, 0] = lo[0] + (r + 1) * cell[0]
        centers[sources, 1] = lo[1]
        z = np.sort(rng.integers(0, 4000, sources.size)) if order != "same" else \
            np.full(sources.size, 7)
        centers[sources, 2] = lo[2] + z * cell[2]
        pick = sources[rng.integers(0, sources.size, n)]
        if order == "ascending":  # sorted by displacement: target minus source
            pick = pick[np.argsort(-centers[pick, 2], kind="stable")]
        src.append(pick)
        tgt.append(np.full(n, target))
    src, tgt = np.concatenate(src), np.concatenate(tgt)
    # pairs at the deepest level reach far in every axis: keys past 64 bits
    far = np.flatnonzero(level == deep)[:2]
    centers[far[0]], centers[far[1 % far.size]] = lo, lo
    corner = np.flatnonzero(level == 1)[:2]
    centers[corner[0]], centers[corner[1]] = hi, lo
    src = np.concatenate([src, [corner[0], far[0], corner[0]]])
    tgt = np.concatenate([tgt, [far[0], corner[0], corner[1]]])
    if order == "any":
        mix = rng.permutation(src.size)
        src, tgt = src[mix], tgt[mix]
    return centers, src.astype(np.int64), tgt.astype(np.int64)


@pytest.mark.parametrize("order", ("same", "ascending", "any"))
@pytest.mark.parametrize("lengths", (RUNS, (3, 16384), (2, 16385, 300), (40000, 260, 5),
                                     (2000000, 40000, 20000, 250)),
                         ids=("edges", "longest", "past", "far past", "a 64th"))
def test_long_runs_match_oracle(cuda_device, oracle, tree, lengths, order):
    import torch

    import yggdrax_b200 as yb

    t, g = tree
    centers, src, tgt = _pairs(t, lengths, order, np.random.default_rng(3))
    geo = g._replace(center=torch.from_numpy(centers).to(cuda_device))
    got = yb.build_grouped_interactions_from_pairs(
        t, geo, torch.from_numpy(src).to(cuda_device), torch.from_numpy(tgt).to(cuda_device))
    cpu = lambda x: x.detach().cpu().numpy()  # noqa: E731
    want = oracle.grouped_from_pairs(src, tgt, cpu(t.node_level), centers, cpu(t.bounds_min),
                                     cpu(t.bounds_max))
    for k, w in want.items():
        np.testing.assert_array_equal(cpu(getattr(got, k)), w, err_msg=k)
    keys = cpu(got.class_keys).astype(np.int64)
    bits = sum(int(x).bit_length() for x in keys.max(0) - keys.min(0))
    assert bits > 64 + 12  # the runs tie in their top words
