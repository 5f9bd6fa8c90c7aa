"""What a program that uses this package asks of it, as cases that can be timed.

A case is a dict of plain values; ``kind`` says which public entry points one
pass goes through:

* ``step``: one step of an N-body program: tree build, node geometry, far and
  near lists from new particle positions;
* ``batched``: the same step for many independent systems at once;
* ``native``: a step whose lists hold the cells of an explicit octree;
* ``moments`` / ``mutual`` / ``grouped``: what such a program computes from a
  tree that it has built.

Point sets are those of ``yggdrax_b200.inputs`` (uniform cube, Plummer sphere,
Plummer clumps), drawn on the GPU.  ``points`` names the snapshot; the seed
gives the order in which its particles are stored, their masses and the unit of
length (a power of two, so the lists keep their lengths from seed to seed).
"""

from __future__ import annotations

import math

import torch

import yggdrax_b200 as yb
from yggdrax_b200 import batch

# A large Plummer sphere has a halo leaf that is near to every other leaf: the
# sizing check of the reference's dense buffers and the dense helper table are
# not for such a tree, so a program that uses one sets both aside.
yb.set_reference_limits(False)
yb.set_dense_neighbor_budget(1 << 28)

_DEV = "cuda"


def listed():
    return [
        # A few thousand bodies with the library's defaults: launches and host
        # work are what such a call costs.
        dict(name="step_cube_4k", kind="step", points=0, dist="cube", tree="radix", n=4000, leaf=8,
             mac="bh", theta=0.5, config=False),
        # The reference's small configuration, with fixed traversal capacities.
        dict(name="step_cube_64k", kind="step", points=1, dist="cube", tree="radix", n=65536,
             leaf=16, mac="dehnen", theta=0.6, config=True),
        # A mid-size galaxy model, a particle count that fits no tile.
        dict(name="step_plummer_1m", kind="step", points=2, dist="plummer", tree="radix", n=1000003,
             leaf=32, mac="dehnen", theta=0.6, config=False),
        # The octree configuration with the Barnes-Hut criterion.
        dict(name="step_octree_4m", kind="step", points=3, dist="plummer", tree="octree", n=4194304,
             leaf=32, mac="bh", theta=0.5, config=False),
        # Clustered points in a fixed-depth octree with local refinement.
        dict(name="step_fixed_clumps_4m", kind="step", points=4, dist="clumps", tree="fixed_octree",
             n=4194304, leaf=32, mac="dehnen", theta=0.6, config=False),
        # The headline workload: 16M Plummer particles on one GPU.
        dict(name="step_plummer_16m", kind="step", points=5, dist="plummer", tree="radix",
             n=16777216, leaf=32, mac="dehnen", theta=0.6, config=False),
        # Many star clusters or halos of uneven size advanced together.
        dict(name="batched_512", kind="batched", points=6, sets=512, leaf=16,
             mac="dehnen", theta=0.6),
        # The upward pass of a fast multipole method, order 4.
        dict(name="moments_256k", kind="moments", points=7, n=262143, leaf=32, order=4),
        # A mutual (momentum-conserving) multipole method's canonical pairs.
        dict(name="mutual_500k", kind="mutual", points=8, n=500000, leaf=32, theta=0.6),
        # Far pairs in displacement classes, for batched translation operators.
        dict(name="grouped_1m", kind="grouped", points=9, n=1048576, leaf=32, theta=0.6),
        # A step of a program that works on the cells of an explicit octree: the
        # tree, far pairs and leaf neighbours between its cells.
        dict(name="native_1m", kind="native", points=10, n=1048576, leaf=32, theta=0.6),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, n))


def draw(rng):
    points = rng.randrange(1000, 1000000)
    kind = rng.choice(("step",) * 6 + ("batched", "moments", "mutual", "grouped", "native"))
    if kind == "step":
        dist, tree = rng.choice((("cube", "radix"), ("plummer", "radix"), ("plummer", "radix"),
                                 ("plummer", "octree"), ("clumps", "fixed_octree")))
        mac, theta = rng.choice((("dehnen", 0.6), ("dehnen", 0.6), ("bh", 0.5),
                                 ("dehnen", 0.5 + 0.01 * rng.randrange(20))))
        top = {"cube": 2000000, "plummer": 16777216, "clumps": 4194304}[dist]
        if mac == "bh" or theta < 0.6:
            top = min(top, 2097152 if dist == "clumps" else 4194304)
        n = _log_int(rng, 4000, top)
        # large particle counts come with large leaves, as in the listed cases
        leaf = rng.choice((8, 16, 32) if n < 100000 else (16, 32) if n < 2000000 else (32,))
        return dict(kind=kind, points=points, dist=dist, tree=tree, n=n, leaf=leaf,
                    mac=mac, theta=theta, config=dist == "cube" and rng.random() < 0.5)
    if kind == "batched":
        return dict(kind=kind, points=points, sets=_log_int(rng, 32, 768),
                    leaf=rng.choice((16, 32)), mac="dehnen", theta=0.6)
    if kind == "moments":
        return dict(kind=kind, points=points, n=_log_int(rng, 20000, 1000000),
                    leaf=rng.choice((16, 32)), order=rng.choice((2, 3, 4)))
    n = _log_int(rng, 20000, 2000000)
    return dict(kind=kind, points=points, n=n, leaf=rng.choice((16, 32)),
                theta=rng.choice((0.5, 0.6, 0.7)))


# ---------------------------------------------------------------------------
# Inputs


def _rand(gen, *shape):
    return torch.rand(shape, generator=gen, device=_DEV, dtype=torch.float64)


def _ball(gen, n, scale, rmax_over_a: float = 20.0):
    """Plummer radii by inversion, truncated at ``rmax_over_a`` scale radii,
    in isotropic directions."""
    top = (1.0 + rmax_over_a ** -2) ** -1.5
    x = _rand(gen, n).clamp_(min=1e-12) * top
    r = scale / torch.sqrt(x ** (-2.0 / 3.0) - 1.0)
    c = 2.0 * _rand(gen, n) - 1.0
    phi = 2.0 * math.pi * _rand(gen, n)
    s = torch.sqrt(1.0 - c * c)
    return torch.stack([r * s * torch.cos(phi), r * s * torch.sin(phi), r * c], dim=1)


def _snapshot(dist: str, n: int, gen):
    if dist == "cube":
        return 2.0 * _rand(gen, n, 3) - 1.0
    if dist == "plummer":
        return _ball(gen, n, 1.0)
    k = 64  # Plummer clumps in a box
    centre = 20.0 * _rand(gen, k, 3) - 10.0
    a = torch.exp(math.log(0.05) + math.log(10.0) * _rand(gen, k))
    which = torch.arange(n, device=_DEV) * k // n
    return centre[which] + _ball(gen, n, a[which])


def _generators(case, seed: int):
    return (torch.Generator(device=_DEV).manual_seed(7919 + int(case["points"])),
            torch.Generator(device=_DEV).manual_seed(104729 + int(seed)))


def _unit(gen) -> float:
    return 2.0 ** int(torch.randint(-3, 4, (1,), generator=gen, device=_DEV))


def _points(case, dist: str, seed: int):
    """``(positions (n, 3), masses (n,))`` float32 on the GPU."""
    of_points, of_seed = _generators(case, seed)
    n = case["n"]
    pos = _snapshot(dist, n, of_points).float()
    order = torch.randperm(n, generator=of_seed, device=_DEV)
    pos = (pos * _unit(of_seed))[order].contiguous()
    if dist == "cube":
        mass = 0.5 + _rand(of_seed, n)
    elif dist == "plummer":  # nearly equal masses
        mass = (1.0 + 0.01 * _rand(of_seed, n)) / n
    else:
        mass = torch.exp(torch.randn(n, generator=of_seed, device=_DEV, dtype=torch.float64))
    return pos, mass.float()


def _set_offsets(case):
    """Set sizes log-uniform in 256 ... 65536."""
    sets = case["sets"]
    gen = torch.Generator().manual_seed(7919 + int(case["points"]))
    u = torch.rand(sets, generator=gen, dtype=torch.float64)
    sizes = torch.exp(math.log(256.0) + u * math.log(256.0)).long().clamp_(256, 65536)
    return torch.cat([torch.zeros(1, dtype=torch.int64), torch.cumsum(sizes, 0)])


def _set_points(case, offsets, seed: int):
    """Every other set a uniform cube, the others Plummer spheres; each set's
    particles in an order of the seed's."""
    of_points, of_seed = _generators(case, seed)
    n = int(offsets[-1])
    sizes = (offsets[1:] - offsets[:-1]).to(_DEV)
    which = torch.repeat_interleave(torch.arange(sizes.numel(), device=_DEV), sizes)
    pos = torch.where((which % 2 == 0)[:, None], _snapshot("cube", n, of_points),
                      _snapshot("plummer", n, of_points)).float()
    order = torch.argsort(which + _rand(of_seed, n))
    pos = (pos * _unit(of_seed))[order].contiguous()
    return pos, (0.5 + _rand(of_seed, n)).float()


def _native_config():
    return yb.DualTreeTraversalConfig(max_pair_queue=1 << 26, process_block=256,
                                      max_interactions_per_node=1 << 20,
                                      max_neighbors_per_leaf=1 << 20)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        pos, mass = _points(case, case["dist"], seed)
        cfg = None
        if case["config"]:
            cfg = yb.DualTreeTraversalConfig(max_pair_queue=1 << 24, process_block=256,
                                             max_interactions_per_node=2048,
                                             max_neighbors_per_leaf=2048)
        return dict(case=case, pos=pos, mass=mass, config=cfg)
    if kind == "batched":
        # the systems and their sizes stay, their particles move
        offsets = _set_offsets(case)
        pos, mass = _set_points(case, offsets, seed)
        return dict(case=case, pos=pos, mass=mass, offsets=offsets)
    if kind == "native":
        pos, mass = _points(case, "clumps", seed)
        return dict(case=case, pos=pos, mass=mass, config=_native_config())
    pos, mass = _points(case, "plummer", seed)
    tree, ps, ms = yb.build_tree(pos, mass, leaf_size=case["leaf"], return_reordered=True)[:3]
    state = dict(case=case, tree=tree, ps=ps, ms=ms)
    if kind == "moments":
        return state
    state["geometry"] = yb.compute_tree_geometry(tree, ps)
    if kind == "mutual":
        total, ni = int(tree.parent.shape[0]), int(tree.left_child.shape[0])
        for side in ("left", "right"):
            full = torch.full((total,), -1, dtype=tree.parent.dtype, device=_DEV)
            full[:ni] = getattr(tree, side + "_child")
            state[side] = full
        # centres of mass lie off the box centres, in spheres that still hold
        # the particles
        g, gen = state["geometry"], _generators(case, seed)[1]
        off = (_rand(gen, total, 3) - 0.5).float()
        state["centers"] = g.center + 0.1 * g.radius[:, None] * off
        state["radii"] = 1.1 * g.radius
        state["cap"] = max(1 << 16, 256 * total)
        return state
    state["far"] = yb.build_interactions_and_neighbors(
        tree, state["geometry"], theta=case["theta"], mac_type="dehnen")[0]
    return state


# ---------------------------------------------------------------------------
# One pass


def _plain(value):
    """A tensor as it is, 64-bit codes as signed integers of the same bits."""
    return value.view(torch.int64) if value.dtype == torch.uint64 else value


def _fields(t):
    return {k: _plain(getattr(t, k)) for k in t._fields if torch.is_tensor(getattr(t, k))}


def _step(state):
    c, pos, mass = state["case"], state["pos"], state["mass"]
    if c["tree"] == "radix":
        tree, ps, ms, inv = yb.build_tree(pos, mass, leaf_size=c["leaf"], return_reordered=True)
    elif c["tree"] == "octree":
        tree, ps, ms, inv = yb.build_octree(pos, mass, leaf_size=c["leaf"], return_reordered=True)
    else:
        tree, ps, ms, inv = yb.build_fixed_depth_octree(
            pos, mass, target_leaf_particles=c["leaf"], return_reordered=True)
    geom = yb.compute_tree_geometry(tree, ps)
    far, near = yb.build_interactions_and_neighbors(
        tree, geom, theta=c["theta"], mac_type=c["mac"], traversal_config=state["config"])
    return dict(tree=_fields(tree.topology), sorted=[ps, ms, inv], geometry=list(geom),
                far=_fields(far),
                near={k: v for k, v in _fields(near).items() if not k.startswith("target_")})


def _batched(state):
    c = state["case"]
    bt = batch.build_trees_batched(state["pos"], state["mass"], state["offsets"],
                                   leaf_size=c["leaf"])
    bg = batch.compute_tree_geometry_batched(bt)
    bi = batch.build_interactions_and_neighbors_batched(bt, bg, theta=c["theta"],
                                                        mac_type=c["mac"])
    tree = {k: _plain(getattr(bt, k)) for k in (
        "inverse_permutation", "particle_indices", "morton_codes", "leaf_starts", "leaf_ends",
        "leaf_codes", "parent", "left_child", "right_child", "left_is_leaf", "right_is_leaf",
        "node_ranges", "node_level", "level_offsets", "nodes_by_level", "num_levels")}
    lists = {k: getattr(bi, k) for k in (
        "node_offsets", "far_counts", "sources", "targets", "target_levels", "near_offsets",
        "near_counts", "neighbors")}
    return dict(tree=tree, sorted=[bt.positions_sorted, bt.masses_sorted],
                geometry=[bg.center, bg.half_extent, bg.radius, bg.max_extent], lists=lists)


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "step":
        return _step(state)
    if kind == "batched":
        return _batched(state)
    if kind == "moments":
        m = yb.compute_tree_multipole_moments(state["tree"], state["ps"], state["ms"],
                                              max_order=c["order"])
        return _fields(m)
    if kind == "mutual":
        return _fields(yb.dual_tree_walk_mutual(
            state["left"], state["right"], state["centers"], state["radii"], c["theta"], 0,
            max_pair_queue=state["cap"], far_cap=state["cap"], near_cap=state["cap"]))
    if kind == "grouped":
        return _fields(yb.build_grouped_interactions(state["tree"], state["geometry"],
                                                     state["far"]))
    tree, ps, ms, inv = yb.build_fixed_depth_octree(
        state["pos"], state["mass"], target_leaf_particles=c["leaf"], return_reordered=True)
    far = yb.build_octree_native_far_pairs(tree, None, theta=c["theta"], mac_type="dehnen",
                                           traversal_config=state["config"])
    near = yb.build_octree_native_neighbor_lists(
        tree, None, theta=c["theta"], mac_type="dehnen", traversal_config=state["config"])
    return dict(tree=_fields(tree.topology), sorted=[ps, ms, inv], far=_fields(far), near={k: v for k, v in _fields(near).items()
                                        if not k.startswith("target_")})


# ---------------------------------------------------------------------------
# What a pass cannot do without

# Directed far and near entries per leaf, as counted on these point sets
# (Dehnen's criterion at theta 0.6, Barnes-Hut at 0.5).
_PER_LEAF = {("cube", "dehnen"): (200, 270), ("cube", "bh"): (100, 150),
             ("plummer", "dehnen"): (390, 620), ("plummer", "bh"): (227, 437),
             ("clumps", "dehnen"): (200, 85), ("clumps", "bh"): (150, 60),
             ("sets", "dehnen"): (174, 303)}


def _per_leaf(dist: str, mac: str, theta: float):
    k = ((0.6 if mac == "dehnen" else 0.5) / theta) ** 3
    return tuple(k * x for x in _PER_LEAF[dist, mac])


def _list_bytes(dist: str, leaves: float, mac: str, theta: float) -> float:
    """Far entries carry source, target and level, near entries one index."""
    far, near = _per_leaf(dist, mac, theta)
    return leaves * (24.0 * min(far, leaves) + 8.0 * min(near, leaves))


def _step_bytes(n: int, leaf: int, dist: str, mac: str, theta: float, tables: int) -> float:
    leaves = -(-n // leaf)
    # read: position, mass; written: both in tree order, code, permutation and
    # its inverse; per node the topology (about 100 bytes), the octree tables
    # where there are any, and the geometry
    return n * (16.0 + 16.0 + 8.0 + 16.0) + 2.0 * leaves * (100.0 + tables + 32.0) + \
        _list_bytes(dist, leaves, mac, theta)


def work(case):
    kind = case["kind"]
    if kind == "step":
        b = _step_bytes(case["n"], case["leaf"], case["dist"], case["mac"], case["theta"],
                        0 if case["tree"] == "radix" else 170)
        leaves = -(-case["n"] // case["leaf"])
        if case["tree"] == "radix" and 8 * leaves * leaves <= 1 << 28:
            b += 8.0 * leaves * leaves  # the dense table of a small tree's neighbours
    elif kind == "batched":
        n = int(_set_offsets(case)[-1])
        b = _step_bytes(n, case["leaf"], "sets", case["mac"], case["theta"], 0)
    elif kind == "moments":
        n, nodes = case["n"], 2 * (-(-case["n"] // case["leaf"])) - 1
        packed = (case["order"] + 1) * (case["order"] + 2) * (case["order"] + 3) // 6
        return dict(bytes=16.0 * n + nodes * (16.0 + 4.0 * (1 + 3 + 3 + 18 + 54 + 162 + packed)),
                    flops=2.0 * n * packed + 2.0 * nodes * packed * packed)
    elif kind == "mutual":
        leaves = -(-case["n"] // case["leaf"])
        # two indices of every pair, far and near; the padded lists come whole
        cap = max(1 << 16, 256 * (2 * leaves - 1))
        b = 2.0 * leaves * 32.0 + 32.0 * cap
    elif kind == "grouped":
        leaves = -(-case["n"] // case["leaf"])
        # a pair is read and written once, with its class; nearly every pair is
        # a class of its own
        far = _per_leaf("plummer", "dehnen", case["theta"])[0]
        b = leaves * far * (16.0 + 24.0 + 40.0)
    else:
        leaves = case["n"] / case["leaf"]
        b = 56.0 * case["n"] + 2.0 * leaves * 300.0 + _list_bytes("clumps", leaves, "dehnen", case["theta"])
    # a handful of operations decide an entry of the lists
    return dict(bytes=b, flops=b)


# ---------------------------------------------------------------------------
# The floating outputs in 64 bits, by plain torch


def _spread(x):
    for shift, keep in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F),
                        (4, 0x10C30C30C30C30C3), (2, 0x1249249249249249)):
        x = (x | (x << shift)) & keep
    return x


def _morton_order(pos):
    """Sorted Morton codes and the stable order, codes as the build defines
    them (float32, 21 bits an axis, a box padded by 5%)."""
    lo, hi = pos.amin(0), pos.amax(0)
    pad = torch.clamp((hi - lo) * torch.tensor(0.05, device=_DEV), min=1e-6)
    lo, hi = lo - pad, hi + pad
    unit = ((pos - lo) / (hi - lo)).clamp_(0.0, 1.0)
    cell = torch.round(unit * 2097151.0).long()
    code = _spread(cell[:, 0]) | (_spread(cell[:, 1]) << 1) | (_spread(cell[:, 2]) << 2)
    return torch.sort(code, stable=True)


def _prefix(a, b):
    """Common leading bits of two 64-bit codes below 2^63 (64 when equal)."""
    x = a ^ b
    n = torch.full_like(x, 64)
    for s in (32, 16, 8, 4, 2, 1):
        big = x >= (1 << s)
        n = torch.where(big, n - s, n)
        x = torch.where(big, x >> s, x)
    return n - x.clamp(max=1)


def _node_leaves(code):
    """First and last leaf under every node of the radix tree over sorted leaf
    codes: internal nodes, then leaves."""
    L = code.numel()
    i = torch.arange(L, device=_DEV)
    if L == 1:
        return i, i

    def delta(a, b):
        ok = (b >= 0) & (b < L)
        s = b.clamp(0, L - 1)
        same = code[a] == code[s]
        d = torch.where(same, 64 + _prefix(a, s), _prefix(code[a], code[s]))
        return torch.where(ok, d, torch.full_like(d, -1))

    k = i[:-1]
    step = torch.sign(delta(k, k + 1) - delta(k, k - 1))
    step = torch.where((k == 0) | (step == 0), torch.ones_like(step), step)
    floor = delta(k, k - step)
    span = torch.zeros_like(k)
    for b in range(L.bit_length(), -1, -1):
        far = delta(k, k + (span + (1 << b)) * step)
        span = torch.where(far > floor, span + (1 << b), span)
    end = k + span * step
    return torch.cat([torch.minimum(k, end), i]), torch.cat([torch.maximum(k, end), i])


def _range_min(x, first, last):
    """Minimum of rows first..last of x (rows, 3) for every query."""
    out = torch.empty((first.numel(), x.shape[1]), dtype=x.dtype, device=x.device)
    length = last - first + 1
    b = 0
    while (1 << b) <= x.shape[0]:
        q = ((length >> b) == 1).nonzero()[:, 0]
        if q.numel():
            out[q] = torch.minimum(x[first[q]], x[last[q] - (1 << b) + 1])
        if x.shape[0] > (1 << b):
            x = torch.cat([torch.minimum(x[: -(1 << b)], x[1 << b:]), x[-(1 << b):]])
        b += 1
    return out


def _radix(pos, leaf: int):
    """Order and, of every node, the particle range [start, end) and leaves."""
    code, order = _morton_order(pos)
    n = code.numel()
    first, last = _node_leaves(code[::leaf])
    return order, first * leaf, torch.clamp((last + 1) * leaf, max=n), first, last


def _boxes(pos, leaf: int):
    """Sorted positions and [centre, half extent, radius, largest extent]."""
    order, _, _, first, last = _radix(pos, leaf)
    p = pos.double()[order]
    n = p.shape[0]
    L = -(-n // leaf)
    q = torch.cat([p, p[-1:].expand(L * leaf - n, 3)]).reshape(L, leaf, 3)
    lo = _range_min(q.amin(1), first, last)
    hi = -_range_min(-q.amax(1), first, last)
    half = torch.clamp(0.5 * (hi - lo), min=1e-6)
    return order, p, [0.5 * (lo + hi), half, half.norm(dim=1), half.amax(1)]


def _combos(order: int):
    return [(i, j, lv - i - j) for lv in range(order + 1) for i in range(lv + 1)
            for j in range(lv + 1 - i)]


def _moments(case, seed):
    pos, mass = _points(case, "plummer", seed)
    perm, start, end, _, _ = _radix(pos, case["leaf"])
    p, m = pos.double()[perm], mass.double()[perm]

    def ranged(w):
        s = torch.cat([torch.zeros(1, dtype=w.dtype, device=_DEV), torch.cumsum(w, 0)])
        return s[end] - s[start]

    total = ranged(m)
    centre = torch.stack([ranged(m * p[:, a]) for a in range(3)], 1) / total[:, None]
    order = case["order"]
    combos = _combos(order)
    raw = {c: ranged(m * p[:, 0] ** c[0] * p[:, 1] ** c[1] * p[:, 2] ** c[2]) for c in combos}
    about = {}
    for c in combos:
        s = torch.zeros_like(total)
        for d in combos:
            if all(x <= y for x, y in zip(d, c)):
                k = math.prod(math.comb(y, x) for x, y in zip(d, c))
                t = k * raw[d]
                for a in range(3):
                    t = t * (-centre[:, a]) ** (c[a] - d[a])
                s = s + t
        about[c] = s

    def tensor(rank):
        t = torch.zeros((total.numel(),) + (3,) * rank, dtype=torch.float64, device=_DEV)
        if rank > order:
            return t
        for flat in range(3 ** rank):
            idx = tuple(flat // 3 ** k % 3 for k in range(rank))
            t[(slice(None),) + idx] = about[tuple(idx.count(a) for a in range(3))]
        return t

    eye = torch.eye(3, dtype=torch.float64, device=_DEV)
    m2, m3, m4 = tensor(2), tensor(3), tensor(4)
    quad = 3.0 * m2 - torch.einsum("naa,ij->nij", m2, eye)
    v = torch.einsum("naak->nk", m3)
    octu = 5.0 * m3 - (torch.einsum("nk,ij->nijk", v, eye) + torch.einsum("nj,ik->nijk", v, eye)
                       + torch.einsum("ni,jk->nijk", v, eye))
    r2 = torch.einsum("naakl->nkl", m4)
    r4 = torch.einsum("naa->n", r2)
    pairs = sum(torch.einsum("nij,kl->n" + s, r2, eye)
                for s in ("ijkl", "ikjl", "iklj", "kijl", "kilj", "klij"))
    deltas = sum(torch.einsum("n,ij,kl->n" + s, r4, eye, eye) for s in ("ijkl", "ikjl", "iklj"))
    hexa = 35.0 * m4 - 5.0 * pairs + deltas
    # about the centre of mass the dipole is zero: no value to be a share of
    return dict(mass=total, center=centre, dipole=None, second_moment=m2, quadrupole=quad,
                third_moment=m3, octupole=octu, fourth_moment=m4, hexadecapole=hexa,
                raw_packed=torch.stack([about[c] for c in combos], 1))


def exact(case, seed):
    kind = case["kind"]
    if kind == "moments":
        return _moments(case, seed)
    if kind == "step" and case["tree"] != "fixed_octree":
        pos, mass = _points(case, case["dist"], seed)
        order, p, geometry = _boxes(pos, case["leaf"])
        return dict(tree=None, sorted=[p, mass.double()[order], None], geometry=geometry,
                    far=None, near=None)
    if kind == "batched":
        offsets = _set_offsets(case)
        pos, mass = _set_points(case, offsets, seed)
        cuts = offsets.tolist()
        parts = [_boxes(pos[a:b], case["leaf"]) for a, b in zip(cuts, cuts[1:])]
        return dict(tree=None, sorted=[torch.cat([x[1] for x in parts]), torch.cat(
            [mass[a:b].double()[x[0]] for x, a, b in zip(parts, cuts, cuts[1:])])],
                    geometry=[torch.cat([x[2][k] for x in parts]) for k in range(4)], lists=None)
    return None
