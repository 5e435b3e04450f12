"""The quantize kernel deals 8-token groups out in equal consecutive shares: shares that begin and end inside a (user, head)
pair, fewer groups than warps, one token, more heads than a block's shares touch.  Bytes and sign bits as the oracle gives
them, norms to 1e-6 (fp32 sums of 128 squares in another order)."""
import pytest
import torch

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T", [(1, 1, 1), (1, 1, 2051), (1, 3, 333), (2, 32, 9), (7, 5, 1), (700, 4, 1), (3, 1, 7000)])
@pytest.mark.parametrize("per_head", [False, True])
def test_shares(B, H, T, per_head):
    from omnistack_rs_b200.kernels.quantize import rotate_quantize_append
    dev = torch.device("cuda:0")
    gen = torch.Generator().manual_seed(B * 100 + H + T)
    x = torch.randn(B, H, T, 128, generator=gen).to(torch.bfloat16)
    cb = torch.sort(torch.randn(H, 16, generator=gen) * 1.2, dim=1).values
    cb = cb if per_head else cb[0].contiguous()
    S = T + 5
    nib = torch.full((B, H, S, 64), 0xAB, dtype=torch.uint8, device=dev)
    qjl = torch.full((B, H, S, 8), 0xCD, dtype=torch.uint8, device=dev)
    norms = torch.full((B, H, S), -1.0, device=dev)
    only = nib.clone()
    rotate_quantize_append(x.to(dev), nib, qjl, norms, 2, cb.to(dev), 9)
    rotate_quantize_append(x.to(dev), only, None, None, 2, cb.to(dev), 9)
    wn, wq, wr = orc.rotate_quantize(x, cb, 9)
    assert torch.equal(nib[:, :, 2:2 + T].cpu(), wn) and torch.equal(qjl[:, :, 2:2 + T].cpu(), wq) and torch.equal(only, nib)
    assert torch.allclose(norms[:, :, 2:2 + T].cpu(), wr, rtol=1e-6, atol=0)
    for part in (slice(0, 2), slice(2 + T, S)):                       # nothing outside the appended rows is touched
        assert (nib[:, :, part] == 0xAB).all() and (qjl[:, :, part] == 0xCD).all() and (norms[:, :, part] == -1.0).all()
