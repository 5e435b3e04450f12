"""Dequantisation on both sides of the rule that picks its work unit (runs of 16 or 64 tokens), with partial last runs behind
full ones in both: the codec's inverse to 1e-5 like every dequantised tensor here."""
import pytest
import torch

import oracle as orc
from tests.helpers import device_us

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,T,with_qjl", [(2, 3, 15, True), (2, 3, 17, True), (1, 2, 129, False), (3000, 4, 2, True), (1501, 8, 1, False),
                                              (1500, 4, 65, True), (1001, 4, 130, True),                  # runs of 64: two and three a pair
                                              (1185, 4, 17, True), (1185, 4, 17, False), (800, 4, 33, False)])   # ... one, partly empty
def test_dequantize_runs(B, H, T, with_qjl):
    from omnistack_rs_b200.kernels.quantize import dequantize_heads
    gen = torch.Generator().manual_seed(B + T)
    nib = torch.randint(0, 256, (B, H, T, 64), generator=gen, dtype=torch.uint8)
    qjl = torch.randint(0, 256, (B, H, T, 8), generator=gen, dtype=torch.uint8)
    norms = torch.rand(B, H, T, generator=gen) * 3
    cb = torch.sort(torch.randn(H, 16, generator=gen), dim=1).values
    got = dequantize_heads(nib.cuda(), qjl.cuda(), norms.cuda(), cb.cuda(), 5, with_qjl).cpu()
    assert (got - orc.dequantize_heads(nib, qjl, norms, cb, 5, with_qjl)).abs().max() <= 1e-5


def test_tokens_just_over_a_short_run():
    """A pair of 17 tokens costs little more per row than one of 16 (1,000,000 rows of codes 97.7 us against 92.1; as a full and an
    almost empty run of 16 tokens 120)."""
    from omnistack_rs_b200.kernels.quantize import dequantize_heads
    us = {}
    for T in (16, 17):
        B = 250000 // T
        nib = torch.zeros(B, 4, T, 64, dtype=torch.uint8, device="cuda")
        qjl, norms = torch.zeros(B, 4, T, 8, dtype=torch.uint8, device="cuda"), torch.zeros(B, 4, T, device="cuda")
        cb = torch.linspace(-2.0, 2.0, 16, device="cuda")
        us[T] = device_us(lambda: dequantize_heads(nib, qjl, norms, cb, 0, False))
    assert us[17] <= 1.15 * us[16], us
