"""The reorder's inverse permutation where its table is as large as 8 of the largest
windows, written in windows, and one entry larger, written in one pass."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,n", [(64, 1 << 26), (64, (1 << 26) + 1), (32, (1 << 27) + 1)])
def test_inverse_at_the_largest_windowed_table(cuda_device, bits, n):
    import torch

    from yggdrax_b200 import _lib as L

    rec = torch.rand(n, 4, device=cuda_device)
    order = torch.randperm(n, device=cuda_device, dtype=torch.int32,
                           generator=torch.Generator(device=cuda_device).manual_seed(1))
    idt = torch.int64 if bits == 64 else torch.int32
    pos, mass = torch.empty(n, 3, device=cuda_device), torch.empty(n, device=cuda_device)
    idx = torch.empty(n, dtype=idt, device=cuda_device)
    inv = torch.full((n,), -1, dtype=idt, device=cuda_device)
    L.check(L.lib().ygx_reorder_packed(L.ptr(rec), L.ptr(order), n, bits, L.ptr(pos), L.ptr(mass),
                                       L.ptr(idx), L.ptr(inv), L.stream_handle(cuda_device)),
            "reorder")
    assert torch.equal(idx, order.to(idt)) and torch.equal(mass, rec[:, 3][order.long()])
    assert torch.equal(inv[order.long()], torch.arange(n, dtype=idt, device=cuda_device))
