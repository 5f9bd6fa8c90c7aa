"""The node kernel of the moments at the edges of its tiles of 16 nodes, on nodes
large enough that a neighbour's or a zero tensor shows: two ranges by turns, so
every node has to equal the first of its kind bit for bit, and those two the
packed coefficients in float64 and the tensors formed from them.

Tolerances.  Packed: the order-k sum of n terms below M (2R)^k, shifted about the
centre, 64 * 2^k * 1.2e-7 * M (2R)^k (the scan's log2 n levels with room).
Tensors: formed from the node's own fp32 coefficients by at most 6 products and 12
sums with factors up to 35, so 64 * 1.2e-7 times 35 times the largest coefficient
of that order."""

from types import SimpleNamespace

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LEVEL = dict(second=2, quad=2, third=3, oct=3, fourth=4, hexa=4)
NAME = dict(second="second_moment", quad="quadrupole", third="third_moment", oct="octupole",
            fourth="fourth_moment", hexa="hexadecapole")


@pytest.mark.parametrize("nodes", (1, 2, 15, 16, 17, 31, 33, 48, 2375))
@pytest.mark.parametrize("order", (1, 2, 3, 4))
def test_every_node_of_every_tile(cuda_device, oracle, nodes, order):
    import torch

    from yggdrax_b200 import inputs
    from yggdrax_b200.dtypes import INDEX_DTYPE
    from yggdrax_b200.tree_moments import _run

    n = 2500
    pos, mass = inputs.uniform_cube(n, 3)
    kinds = np.array([[0, n - 1], [400, 1233]])
    ranges = kinds[np.arange(nodes) % 2]
    topo = SimpleNamespace(
        parent=torch.zeros(nodes, dtype=INDEX_DTYPE, device=cuda_device),
        node_ranges=torch.from_numpy(ranges).to(INDEX_DTYPE).to(cuda_device))
    out = _run(topo, torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device),
               order, None, True)
    for k, v in out.items():
        for kind in range(min(2, nodes)):
            rows = v[kind::2].reshape((nodes - kind + 1) // 2, -1)
            assert torch.equal(rows, rows[:1].expand_as(rows)), (k, kind)
    got = {k: v.cpu().numpy() for k, v in out.items()}
    combos = oracle._combos(order)
    level = np.array([sum(c) for c in combos])
    for v in range(min(2, nodes)):
        a, b = kinds[v]
        c = got["center"][v].astype(np.float64)
        w, d = mass[a:b + 1].astype(np.float64), pos[a:b + 1].astype(np.float64) - c
        want = np.array([(w * d[:, 0] ** i * d[:, 1] ** j * d[:, 2] ** k).sum()
                         for i, j, k in combos])
        atol = 64 * 1.2e-7 * w.sum() * 2.0 ** level * 2.0 ** level
        assert (np.abs(got["packed"][v] - want) <= atol).all()
        packed = got["packed"][v:v + 1]
        tensors = oracle._tensors_from_packed(packed, got["center"][v:v + 1], order)
        for k, lv in LEVEL.items():
            t = got[k][v]
            if lv > order:
                assert not t.any(), k
                continue
            top = np.abs(packed[0][level == lv]).max()
            assert top > 1e-3 * w.sum()
            assert (np.abs(t - tensors[NAME[k]][0]) <= 64 * 1.2e-7 * 35 * top).all(), k
