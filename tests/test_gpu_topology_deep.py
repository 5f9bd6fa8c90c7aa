"""The topology build on trees deeper than the 64 level bins: codes that part one
bit a level, with ties below the last -- nodes_by_level by two digits, and the level
tables of levels 0..63 -- against a restatement of the level rules on the parents
that the build itself returns, and of the parents on the children."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def build(dev, codes):
    import torch

    from yggdrax_b200 import _lib as L
    from yggdrax_b200.dtypes import INDEX_BITS, INDEX_DTYPE

    lib, n = L.lib(), len(codes)
    c = torch.from_numpy(np.asarray(codes, np.uint64).view(np.int64)).to(dev).view(torch.uint64)
    starts = torch.arange(n, dtype=INDEX_DTYPE, device=dev)
    e = lambda k, dt=INDEX_DTYPE: torch.zeros(k, dtype=dt, device=dev)  # noqa: E731
    total, ni, i32 = 2 * n - 1, n - 1, torch.int32
    out = dict(parent=e(total), left=e(ni), right=e(ni), lil=e(ni, torch.bool),
               ril=e(ni, torch.bool), ranges=e(2 * total), level=e(total), level_offsets=e(65),
               nbl=e(total), num_levels=e(1), parent32=e(total, i32), left32=e(total, i32),
               right32=e(total, i32), level32=e(total, i32), nbl32=e(total, i32),
               flags=e(1, i32))
    ws = L.workspace(lib.ygx_topology_workspace_size(n), dev)
    run = lambda: lib.ygx_build_topology(  # noqa: E731
        L.ptr(c), L.ptr(starts), L.ptr(starts + 1), n, INDEX_BITS,
        *[L.ptr(t) for t in out.values()], L.ptr(ws), ws.numel(), L.stream_handle(dev))
    assert run() == 0
    return {k: t.cpu().numpy() for k, t in out.items()}, run


def doubled(parent):
    """Levels by synchronous pointer doubling."""
    n = parent.shape[0]
    up = np.where(parent < 0, np.arange(n), parent)
    d = (parent >= 0).astype(np.int32)
    for _ in range(int(n).bit_length() + 1):
        d, up = (d + d[up]).astype(np.int32), up[up]
    return d


@pytest.mark.parametrize("ties", (1, 9, 10, 300, 5000, 200000))
@pytest.mark.parametrize("base", (0, (1 << 63) - 1))
def test_levels_past_the_bins(cuda_device, ties, base):
    codes = np.sort(np.array([base] * ties + [base ^ (1 << j) for j in range(63)], np.uint64))
    got = build(cuda_device, codes)[0]
    n = codes.size
    total, ni = 2 * n - 1, n - 1
    claim = np.full(total, -1, np.int64)
    np.maximum.at(claim, got["left"], np.arange(ni))
    np.maximum.at(claim, got["right"], np.arange(ni) + ni)
    parent = np.where(claim < 0, -1, np.where(claim >= ni, claim - ni, claim))
    assert np.array_equal(got["parent"], parent) and np.array_equal(got["parent32"], parent)
    level = doubled(parent)
    if base == 0:
        assert level.max() == (63 if ties == 1 else 65)
    assert np.array_equal(got["level"], level) and np.array_equal(got["level32"], level)
    order = np.argsort(level, kind="stable")
    assert np.array_equal(got["nbl"], order) and np.array_equal(got["nbl32"], order)
    held = np.bincount(level, minlength=64)[:64]
    assert np.array_equal(got["level_offsets"], np.concatenate([[0], np.cumsum(held)]))
    assert int(got["num_levels"][0]) == min(64, int(level.max()) + 1)
