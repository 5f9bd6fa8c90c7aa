"""The one-launch topology build at the sizes and shapes where its stages can
go wrong: trees of a few nodes, of one chunk (512 nodes) per CTA and of several
chunks, and tied leaf codes -- parent chains too long to climb, cycles, levels
past the 64 bins -- against the oracle, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = ("parent", "left_child", "right_child", "left_is_leaf", "right_is_leaf", "node_ranges",
          "node_level", "level_offsets", "nodes_by_level", "num_levels")


def _points(kind, n):
    from yggdrax_b200 import inputs

    pos, mass = inputs.uniform_cube(n, n)
    if kind == "ties":      # a tenth of the points on one spot
        pos[: n // 10] = pos[0]
    elif kind == "same":    # every code tied
        pos[:] = pos[0]
        pos[-1] += 1.0      # (with an extent)
    elif kind == "line":    # clustered towards a corner: deep trees
        pos[:] = (2.0 ** -np.linspace(0, 20, n))[:, None].astype(np.float32)
    return pos, mass


@pytest.mark.parametrize("kind", ("cube", "ties", "same", "line"))
@pytest.mark.parametrize("n,leaf", [(2, 1), (3, 1), (256, 1), (257, 1), (5000, 1), (40000, 3),
                                    (310000, 1)])
def test_topology_matches_oracle(cuda_device, oracle, kind, n, leaf):
    import torch

    import yggdrax_b200 as yb

    pos, mass = _points(kind, n)
    P, M = torch.from_numpy(pos).to(cuda_device), torch.from_numpy(mass).to(cuda_device)
    got = yb.build_tree(P, M, leaf_size=leaf, return_reordered=True)[0].topology
    want = oracle.build_tree(pos, mass, leaf_size=leaf)
    for f in FIELDS:
        g = getattr(got, f).cpu().numpy()
        w = np.asarray(getattr(want, f))
        assert np.array_equal(g.astype(np.int64), w.astype(np.int64).reshape(g.shape)), f
