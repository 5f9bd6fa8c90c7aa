"""The reorder's inverse permutation at the edges of its dispatch: in one pass
up to 16 MB, in up to 8 windows of 16 MB, then in larger windows."""
import pytest

pytestmark = pytest.mark.gpu

W64 = (16 << 20) // 8  # entries of one window, 64-bit indices


@pytest.mark.parametrize("packed", [True, False])
@pytest.mark.parametrize("bits,n", [
    (64, 1), (64, 1023), (64, W64), (64, W64 + 1), (64, 3 * W64 - 1), (64, 8 * W64),
    (64, 8 * W64 + 7), (32, 2 * W64), (32, 2 * W64 + 1), (32, 5 * W64 + 3),
])
def test_reorder_and_inverse(cuda_device, packed, bits, n):
    import torch

    from yggdrax_b200 import _lib as L

    lib = L.lib()
    g = torch.Generator(device=cuda_device).manual_seed(n)
    rec = torch.rand(n, 4, device=cuda_device, generator=g)
    order = torch.randperm(n, device=cuda_device, generator=g)
    o32 = order.to(torch.int32)
    idt = torch.int64 if bits == 64 else torch.int32
    pos = torch.empty(n, 3, device=cuda_device)
    mass = torch.empty(n, device=cuda_device)
    idx = torch.empty(n, dtype=idt, device=cuda_device)
    inv = torch.full((n,), -1, dtype=idt, device=cuda_device)
    st = L.stream_handle(rec.device)
    out = (L.ptr(pos), L.ptr(mass), L.ptr(idx), L.ptr(inv), st)
    if packed:
        L.check(lib.ygx_reorder_packed(L.ptr(rec), L.ptr(o32), n, bits, *out), "reorder")
    else:
        p, m = rec[:, :3].contiguous(), rec[:, 3].contiguous()
        L.check(lib.ygx_reorder(L.ptr(p), L.ptr(m), L.ptr(o32), n, bits, *out), "reorder")
    assert torch.equal(pos, rec[order, :3]) and torch.equal(mass, rec[order, 3])
    assert torch.equal(idx, order.to(idt))
    assert torch.equal(inv[order], torch.arange(n, dtype=idt, device=cuda_device))
