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
