"""Which walk forms a batch's lists: the per-target walk for small forests and
where lists of some length are expected, the generation walk for many small sets,
wide openings and short lists met before, for forests past the slots' range and for
sets without pairs."""

from types import SimpleNamespace

import pytest


def _route(monkeypatch, sets, nodes_per_set, leaf=16, mac="dehnen", theta=0.6, scale=1.0,
           entries=0):
    from yggdrax_b200 import batch as B

    taken = []

    def lists(name):
        def form(*args):
            taken.append(name)
            return SimpleNamespace(stats=dict(far_total=entries // 2,
                                              near_total=entries - entries // 2))
        return form

    monkeypatch.setattr(B, "_target_lists_batched", lists("target"))
    monkeypatch.setattr(B, "_log_lists_batched", lists("log"))
    forest = SimpleNamespace(num_sets=sets, total_nodes=sets * nodes_per_set, leaf_size=leaf,
                             total_leaves=sets * (nodes_per_set + 1) // 2)
    B.build_interactions_and_neighbors_batched(forest, None, theta=theta, mac_type=mac,
                                               dehnen_radius_scale=scale)
    return taken[-1]


@pytest.fixture(autouse=True)
def no_hints(monkeypatch):
    from yggdrax_b200 import batch as B

    monkeypatch.setattr(B, "_ENTRIES_HINTS", {})


@pytest.mark.parametrize("sets,nodes,kw,target", [
    (1, 1, {}, False), (1000, 1, {}, False),           # no pairs
    (1, 3, {}, True), (512, 1439, {}, True),
    (666, 37, {}, True), (5000, 37, {}, True),         # a small forest
    (26666, 37, {}, False), (20000, 37, {}, False), (8000, 125, {}, False),
    (1500, 375, {}, True), (8000, 375, {}, True),
    (999, 1499, dict(leaf=4), True), (999, 1499, dict(leaf=4, theta=1.2), False),
    (999, 1499, dict(leaf=4, theta=1.2, scale=2.0), True),
    (999, 1499, dict(leaf=1), False), (2000, 999, dict(mac="bh", theta=0.5), True),
    (2000, 999, dict(mac="bh", theta=0.9), False), (2000, 999, dict(theta=0.0), True),
    (1, (1 << 23) - 1, {}, True), (1, (1 << 23) + 1, {}, False),
])
def test_route(monkeypatch, sets, nodes, kw, target):
    assert _route(monkeypatch, sets, nodes, **kw) == ("target" if target else "log")


def test_short_lists_are_remembered(monkeypatch):
    forest = (999, 1499)
    assert _route(monkeypatch, *forest, entries=3 * 999 * 1499) == "target"
    assert _route(monkeypatch, *forest, entries=120 * 999 * 1499) == "log"
    assert _route(monkeypatch, *forest) == "target"
