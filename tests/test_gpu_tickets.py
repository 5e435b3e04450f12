"""Split-K calls with more work items than warps: a warp that has served its first item draws tickets for the next ones from a
counter (one per kv head where codebooks are per head), cleared by the preparation launch or by a memset.  A counter that is
not cleared, or not the head's own, skips or repeats items.  Every call runs twice over one workspace, with other queries the
second time, so that a skipped item leaves the first call's partial state behind."""
import pytest
import torch

import oracle as orc
from tests.test_gpu_attention import make_cache, to_dev, attn_mod

pytestmark = pytest.mark.gpu

ATOL = 3e-3          # the attention parity tests' budget


@pytest.mark.parametrize("prep", ["0", "1"])
@pytest.mark.parametrize("B,Hq,Hkv,per_head,n_splits,rank", [
    (3, 8, 8, True, 100, 0),         # 300 items per head on 18 x 12 warps, one column
    (3, 16, 8, True, 100, 0),        # ... two columns: ragged users longest first with the preparation launch
    (2, 16, 8, False, 120, 0),       # 1,920 items on 148 x 12 warps, one counter
    (3, 16, 8, True, 200, 0),        # two to three rounds of items
    (3, 16, 8, True, 100, 16),       # the folded query update's kernels
    (2, 8, 8, False, 120, 16),
])
def test_more_items_than_warps(B, Hq, Hkv, per_head, n_splits, rank, prep, monkeypatch):
    monkeypatch.setenv("OMNI_QATTN_KERNEL", "mma")
    monkeypatch.setenv("OMNI_QATTN_PREP", prep)
    monkeypatch.setenv("OMNI_LORA_FOLD", "1")
    fa = attn_mod()
    dev = torch.device("cuda:0")
    S = 2500
    kn, kq, kr, vn, cb, gen = make_cache(B, Hkv, S, seed=B + n_splits, user_id=6, per_head=per_head)
    lens = torch.tensor([S, 1300, 700][:B], dtype=torch.int32)
    cache = to_dev(dev, kn, kq, kr, vn, cb)
    x = torch.randn(B, 1, 128, generator=gen)
    la, lb = torch.randn(2, 16, 128, generator=gen) * 0.04, torch.randn(2, Hq * 128, 16, generator=gen) * 0.1
    idx = torch.tensor([1, -1, 0][:B], dtype=torch.int32)
    lora = dict(x=x.to(dev), lora_a=la.to(dev), lora_b=lb.to(dev), lora_indices=idx.to(dev), lora_alpha=0.3) if rank else {}
    for _ in range(2):
        q = torch.randn(B, Hq, 1, 128, generator=gen).to(torch.bfloat16)
        got = fa.omni_attn(q.to(dev), *cache, user_id=6, seq_lens=lens.to(dev), n_splits=n_splits, **lora).cpu()
        q_eff = orc.apply_lora_to_q(q, x, la, lb, idx, 0.3) if rank else q
        for b, n in enumerate(lens.tolist()):
            want = orc.decode_attention(q_eff[b:b + 1], kn[b:b + 1, :, :n], kq[b:b + 1, :, :n], kr[b:b + 1, :, :n], vn[b:b + 1, :, :n], cb, 6)
            assert (got[b:b + 1] - want).abs().max() <= ATOL, b
