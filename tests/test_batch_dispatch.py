"""Which walk forms a batch's lists: the per-target walk for small forests and
for sets of some size, the generation walk for many small sets, for forests past
the slots' range and for sets without pairs."""

from types import SimpleNamespace

import pytest


@pytest.mark.parametrize("sets,nodes_per_set,target", [
    (1, 1, False), (1000, 1, False),           # no pairs
    (1, 3, True), (512, 1439, True),
    (666, 37, True), (5000, 37, True),         # a small forest
    (26666, 37, False), (20000, 37, False), (8000, 125, False),
    (1333, 375, True), (8000, 375, True),
    (1, (1 << 23) - 1, True), (1, (1 << 23) + 1, False),
])
def test_route(monkeypatch, sets, nodes_per_set, target):
    from yggdrax_b200 import batch as B

    taken = []
    monkeypatch.setattr(B, "_target_lists_batched", lambda *a: taken.append("target") or "lists")
    monkeypatch.setattr(B, "_log_lists_batched", lambda *a: taken.append("log") or "lists")
    forest = SimpleNamespace(num_sets=sets, total_nodes=sets * nodes_per_set,
                             total_leaves=sets * (nodes_per_set + 1) // 2)
    assert B.build_interactions_and_neighbors_batched(forest, None) == "lists"
    assert taken == ["target" if target else "log"]
