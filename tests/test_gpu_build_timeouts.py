"""A grid barrier of the topology builds that gives up (wait limit 0) is
reported: in the flags word that the build reads back, and in the status word
of the workspace, whatever the two held before.  Nothing uses the tables of
such a build here."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class spin_limit:
    """The limit of the device-side waits inside a with block."""

    def __init__(self, value):
        from yggdrax_b200 import _lib as L

        self.lib, self.knob, self.value = L.lib(), L.TUNE["spin_limit"], value

    def __enter__(self):
        old = np.zeros(1, np.int32)
        assert self.lib.ygx_tune_get(self.knob, old.ctypes.data) == 0
        self.old = int(old[0])
        assert self.lib.ygx_tune_set(self.knob, self.value) == 0

    def __exit__(self, *exc):
        assert self.lib.ygx_tune_set(self.knob, self.old) == 0


def _topology(dev, leaves, dirt):
    """(flags word, status word) of a build on a workspace filled with dirt."""
    import torch

    from yggdrax_b200 import _lib as L
    from yggdrax_b200.dtypes import INDEX_BITS, INDEX_DTYPE

    lib, st = L.lib(), L.stream_handle(dev)
    codes = (torch.arange(leaves, dtype=torch.int64, device=dev) << 20).view(torch.uint64)
    starts = torch.arange(leaves, dtype=INDEX_DTYPE, device=dev)
    e = lambda n, dt=INDEX_DTYPE: torch.zeros(n, dtype=dt, device=dev)  # noqa: E731
    total, ni, i32 = 2 * leaves - 1, leaves - 1, torch.int32
    out = [e(total), e(ni), e(ni), e(ni, torch.bool), e(ni, torch.bool), e(2 * total), e(total),
           e(65), e(total), e(1), e(total, i32), e(total, i32), e(total, i32), e(total, i32),
           e(total, i32), torch.full((1,), dirt, dtype=i32, device=dev)]
    ws = torch.full((int(lib.ygx_topology_workspace_size(leaves)),), dirt & 0xff,
                    dtype=torch.uint8, device=dev)
    rc = lib.ygx_build_topology(L.ptr(codes), L.ptr(starts), L.ptr(starts + 1), leaves,
                                INDEX_BITS, *[L.ptr(t) for t in out], L.ptr(ws), ws.numel(), st)
    assert rc == 0
    return int(out[-1].item()), L.read_status(ws)


@pytest.mark.parametrize("dirt", (0, -1))
def test_topology_reports_a_barrier_that_gave_up(cuda_device, dirt):
    from yggdrax_b200 import _lib as L

    assert _topology(cuda_device, 40000, dirt) == (0, 0)
    with spin_limit(0):
        for _ in range(5):  # 157 CTAs: some always wait
            flags, status = _topology(cuda_device, 40000, dirt)
            assert flags & L.FLAG_TIMEOUT and status & L.FLAG_TIMEOUT
    assert _topology(cuda_device, 40000, dirt) == (0, 0)


def test_batched_topology_reports_a_barrier_that_gave_up(cuda_device):
    """In every set's flags, which the walks over the forest read.  (The
    workspace is zeroed: the sort inside, whose waits give up too, then leaves
    no id out of range.)"""
    import torch

    from yggdrax_b200 import _lib as L
    from yggdrax_b200.dtypes import INDEX_BITS, INDEX_DTYPE

    lib, dev = L.lib(), cuda_device
    S, per = 5, 8000
    leaves = S * per
    total, ni, i32 = 2 * leaves - S, leaves - S, torch.int32
    codes = (torch.arange(per, dtype=torch.int64, device=dev) << 20).repeat(S).view(torch.uint64)
    starts = torch.arange(per, dtype=INDEX_DTYPE, device=dev).repeat(S)
    leaf_off = torch.arange(S + 1, dtype=torch.int64, device=dev) * per
    leaf_seg = torch.arange(S, dtype=i32, device=dev).repeat_interleave(per)
    e = lambda n, dt=INDEX_DTYPE: torch.zeros(n, dtype=dt, device=dev)  # noqa: E731
    out = [e(total), e(ni), e(ni), e(ni, torch.bool), e(ni, torch.bool), e(2 * total), e(total),
           e(65 * S), e(total), e(S)] + [e(total, i32) for _ in range(8)] + \
        [e(leaves, i32), e(S, i32), e(1, i32)]

    def run():
        ws = torch.zeros(int(lib.ygx_batch_topology_workspace_size(leaves, S)),
                         dtype=torch.uint8, device=dev)
        rc = lib.ygx_batch_build_topology(
            L.ptr(codes), L.ptr(starts), L.ptr(starts + 1), L.ptr(leaf_off), L.ptr(leaf_seg), S,
            leaves, INDEX_BITS, *[L.ptr(t) for t in out], L.ptr(ws), ws.numel(),
            L.stream_handle(dev))
        assert rc == 0
        return out[-2].tolist(), int(out[-1].item())

    assert run() == ([0] * S, 0)
    with spin_limit(0):
        for _ in range(5):
            sets, union = run()
            assert union & L.FLAG_TIMEOUT and all(f & L.FLAG_TIMEOUT for f in sets)
    assert run() == ([0] * S, 0)


def test_lists_of_a_forest_whose_build_gave_up_are_refused(cuda_device):
    import torch

    from yggdrax_b200 import _lib as L
    from yggdrax_b200 import batch as B

    off = np.arange(21, dtype=np.int64) * 700
    pos = torch.rand(int(off[-1]), 3, generator=torch.Generator().manual_seed(2)).to(cuda_device)
    bt = B.build_trees_batched(pos, torch.ones_like(pos[:, 0]), off, leaf_size=8)
    bg = B.compute_tree_geometry_batched(bt)
    B.build_interactions_and_neighbors_batched(bt, bg, theta=0.5, mac_type="bh")
    bt.seg_flags.bitwise_or_(L.FLAG_TIMEOUT)
    assert B._target_lists_batched(bt, bg, 0.5, "bh", 1.0) is None
    with pytest.raises(L.YgxError):
        B._log_lists_batched(bt, bg, 0.5, "bh", 1.0)
    with pytest.raises(L.YgxError):
        B.build_interactions_and_neighbors_batched(bt, bg, theta=0.5, mac_type="bh")
