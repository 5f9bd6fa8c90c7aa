"""The batched topology's workspace holds every node of the forest, also where
every set is a single leaf (as many nodes as sets)."""

import pytest


@pytest.mark.parametrize("sets,per_set", [(1, 1), (1000, 1), (65536, 1), (1000, 2), (3, 70000)])
def test_batched_topology_workspace_holds_the_forest(sets, per_set):
    from yggdrax_b200 import _lib as L

    leaves = sets * per_set
    nodes = 2 * leaves - sets
    # per node: claim, two root and two depth words, an id (4 bytes each) and
    # a sort key with its sorted copy (8 bytes each); per set its levels' counts
    # and its deepest level
    need = nodes * (6 * 4 + 2 * 8) + sets * (64 * 4 + 4)
    assert L.lib().ygx_batch_topology_workspace_size(leaves, sets) >= need
