"""Dequantisation on both sides of the rule that picks its work unit (runs of 16 or 64 tokens), with partial last runs: the
codec's inverse to 1e-5 like every dequantised tensor here."""
import pytest
import torch

import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,with_qjl", [(2, 3, 15, True), (2, 3, 17, True), (1, 2, 129, False), (3000, 4, 2, True), (1501, 8, 1, False)])
def test_dequantize_runs(B, H, T, with_qjl):
    from omnistack_rs_b200.kernels.quantize import dequantize_heads
    gen = torch.Generator().manual_seed(B + T)
    nib = torch.randint(0, 256, (B, H, T, 64), generator=gen, dtype=torch.uint8)
    qjl = torch.randint(0, 256, (B, H, T, 8), generator=gen, dtype=torch.uint8)
    norms = torch.rand(B, H, T, generator=gen) * 3
    cb = torch.sort(torch.randn(H, 16, generator=gen), dim=1).values
    got = dequantize_heads(nib.cuda(), qjl.cuda(), norms.cuda(), cb.cuda(), 5, with_qjl).cpu()
    assert (got - orc.dequantize_heads(nib, qjl, norms, cb, 5, with_qjl)).abs().max() <= 1e-5
