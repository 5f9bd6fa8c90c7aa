"""The unordered per-target walks keep no room for sorting the chunks' records,
which only the ordered walk does: their workspace grows by a record's key and
its chunk alone."""

import numpy as np
import pytest


def _size(fn, caps, *tail):
    return fn(1001, 501, np.asarray(caps, np.int64).ctypes.data, *tail)


@pytest.mark.parametrize("which", ("tree", "forest"))
def test_unordered_workspace_per_record(which):
    from yggdrax_b200 import _lib as L

    lib = L.lib()
    fn, tail = ((lib.ygx_target_walk_workspace_size, (0,)) if which == "tree"
                else (lib.ygx_batch_target_walk_workspace_size, ()))
    base, more = [1 << 16] * 8, 1 << 20
    near = base[:5] + [base[5] + more] + base[6:]
    assert _size(fn, near, *tail) - _size(fn, base, *tail) == more * (8 + 16)
    if which == "tree":  # the ordered walk sorts them
        assert _size(fn, near, 1) - _size(fn, base, 1) > more * (8 + 16 + 4 + 8 + 4 + 8)
