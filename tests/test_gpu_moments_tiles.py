"""Moments at the edges of their kernels' tiles (2048 particles of the prefix
sums, 16 nodes of the node kernel) against the oracle's formulas in float64,
and what an infinite mass does.

Tolerance: the fp32 prefixes are differenced, so an order-k sum is off by a
few (log2 n, the depth of the scan) eps of the whole system's sum of order k,
and the shift to the centre adds up to 2^k such terms:
64 * 2^k * 1.2e-7 * M (2 R)^k covers 16 levels with a factor of 4."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ORDER = dict(mass=0, second_moment=2, quadrupole=2, third_moment=3, octupole=3, fourth_moment=4,
             hexadecapole=4)


@pytest.mark.parametrize("n,leaf", [(1, 4), (8, 8), (9, 8), (64, 8), (65, 8), (72, 8), (2047, 16),
                                    (2048, 16), (2049, 16), (4097, 4)])
@pytest.mark.parametrize("order", (0, 1, 2, 3, 4))
def test_moments_at_tile_edges(cuda_device, oracle, n, leaf, order):
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(n, 3)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    t, ps, ms = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[:3]
    centers = yb.compute_tree_geometry(t, ps).center
    got = yb.compute_tree_multipole_moments(t, ps, ms, expansion_centers=centers, max_order=order)
    r = t.node_ranges.cpu().numpy()
    p, m = ps.cpu().numpy().astype(np.float64), ms.cpu().numpy().astype(np.float64)
    c = centers.cpu().numpy().astype(np.float64)
    want = {k: np.zeros(getattr(got, k).shape) for k in ORDER}
    packed = np.zeros(got.raw_packed.shape)
    combos = oracle._combos(order)
    for v in range(r.shape[0]):
        d, w = p[r[v, 0]:r[v, 1] + 1] - c[v], m[r[v, 0]:r[v, 1] + 1]
        for q, (i, j, k) in enumerate(combos):
            packed[v, q] = (w * d[:, 0] ** i * d[:, 1] ** j * d[:, 2] ** k).sum()
    want.update({k: x for k, x in oracle._tensors_from_packed(packed, c, order).items()
                 if k in ORDER})
    scale = m.sum()
    for k, lv in ORDER.items():
        atol = 64 * 2.0 ** lv * 1.2e-7 * scale * 2.0 ** lv * (35 if lv == 4 else 5)
        np.testing.assert_allclose(getattr(got, k).cpu().numpy(), want[k], rtol=1e-5, atol=atol,
                                   err_msg=k)
    np.testing.assert_allclose(got.raw_packed.cpu().numpy(), packed, rtol=1e-5,
                               atol=64 * 4.0 ** order * 1.2e-7 * scale)


def test_infinite_mass_reaches_every_coefficient(cuda_device):
    """0 * inf counts in the dense stencil: no coefficient of a node whose
    sums are not finite may come out finite."""
    import torch

    import yggdrax_b200 as yb
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(300, 3)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    t, ps, ms = yb.build_tree(P, M, leaf_size=8, return_reordered=True)[:3]
    ms = ms.clone()
    ms[7] = float("inf")
    r = yb.compute_tree_multipole_moments(t, ps, ms, max_order=4)
    bad = ~torch.isfinite(r.mass)
    assert bool(bad.any())
    assert not bool(torch.isfinite(r.raw_packed[bad]).any())
