"""Codebooks that the fp16 tables cannot hold (a centroid of magnitude 8 or more): the warp-level grid serves the call in fp32,
with every feature the call may have, and about as fast as the fp32 kernel launched for it.

Tolerance.  Both sides sum in fp32.  Scores reach about 10 here; 192 additions round them by at most 192 * 2^-24 * 10 = 1.1e-4,
and a score error of d moves an output by at most 2 d max|centroid| = 32 d.  A tenth of that worst case is asserted, 4e-4."""
import pytest
import torch

import oracle as orc
from tests.helpers import device_us
from tests.test_gpu_attention import make_cache, to_dev, attn_mod

pytestmark = pytest.mark.gpu

ATOL = 4e-4


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch.device("cuda:0")


def wide_cache(B, Hkv, S, seed, per_head):
    kn, kq, kr, vn, cb, gen = make_cache(B, Hkv, S, seed=seed, user_id=6, per_head=per_head)
    return kn, kq, kr, vn, cb * (15.5 / float(cb.abs().max())), gen


@pytest.mark.parametrize("kernel", ["mma", "lane"])
@pytest.mark.parametrize("Hq,Hkv,T,S,n_splits,per_head", [(8, 8, 1, 300, 1, True), (8, 2, 1, 37, 1, False), (6, 2, 3, 130, 3, True),
                                                          (4, 1, 1, 1000, 7, False), (3, 3, 1, 8, 2, True)])
def test_wide_matches_oracle(dev, kernel, Hq, Hkv, T, S, n_splits, per_head, monkeypatch):
    monkeypatch.setenv("OMNI_QATTN_KERNEL", kernel)
    fa = attn_mod()
    kn, kq, kr, vn, cb, gen = wide_cache(4, Hkv, S, S + T, per_head)
    q = (torch.randn(4, Hq, T, 128, generator=gen) * 0.2).to(torch.bfloat16)
    lens = torch.tensor([S, 0, max(1, S - 3), (S + 1) // 2], dtype=torch.int32)
    d = to_dev(dev, q, kn, kq, kr, vn, cb)
    paired = d[4].clone()
    fa.pair_v_rows(paired, 0, lens.to(dev).to(torch.int64))
    for with_qjl in (True, False):
        got = fa.omni_attn(*d, user_id=6, seq_lens=lens.to(dev), n_splits=n_splits, with_qjl=with_qjl)
        assert torch.equal(got, fa.omni_attn(*d[:4], paired, d[5], user_id=6, seq_lens=lens.to(dev), n_splits=n_splits, with_qjl=with_qjl, v_paired=True))
        for b, n in enumerate(lens.tolist()):
            if n == 0:
                assert not got[b].any()
                continue
            want = orc.decode_attention(q[b:b + 1], kn[b:b + 1, :, :n], kq[b:b + 1, :, :n], kr[b:b + 1, :, :n], vn[b:b + 1, :, :n], cb, 6, None, with_qjl)
            assert (got[b:b + 1].cpu() - want).abs().max() <= ATOL, (b, with_qjl)


@pytest.mark.parametrize("kernel", ["mma", "lane"])
@pytest.mark.parametrize("Hq,Hkv,T,hid,rank", [(8, 8, 1, 128, 16), (8, 2, 1, 128, 32), (4, 1, 1, 128, 24), (6, 2, 1, 100, 6), (4, 2, 3, 256, 40)])
def test_wide_with_the_query_update(dev, kernel, Hq, Hkv, T, hid, rank, monkeypatch):
    """The update folded into the fp32 code equals the separate launch bit for bit."""
    monkeypatch.setenv("OMNI_QATTN_KERNEL", kernel)
    fa = attn_mod()
    from omnistack_rs_b200 import _lib
    B = 5
    kn, kq, kr, vn, cb, gen = wide_cache(B, Hkv, 150, rank, True)
    q = (torch.randn(B, Hq, T, 128, generator=gen) * 0.2).to(torch.bfloat16)
    x = torch.randn(B, T, hid, generator=gen)
    la = torch.randn(5, rank, hid, generator=gen) * (0.5 / hid ** 0.5)
    lb = torch.randn(5, Hq * 128, rank, generator=gen) * (0.2 / rank ** 0.5)
    idx = torch.tensor([-1, 0, 4, 2, 2], dtype=torch.int32)
    cache = to_dev(dev, kn, kq, kr, vn, cb)
    lora = dict(x=x.to(dev), lora_a=la.to(dev), lora_b=lb.to(dev), lora_indices=idx.to(dev), lora_alpha=0.3)
    want = orc.decode_attention(orc.apply_lora_to_q(q, x, la, lb, idx, 0.3), kn, kq, kr, vn, cb, 6)
    for n_splits in (1, 3):
        got = []
        for flag in ("1", "0"):
            monkeypatch.setenv("OMNI_LORA_FOLD", flag)
            got.append(fa.omni_attn(q.to(dev), *cache, user_id=6, n_splits=n_splits, **lora))
        assert torch.equal(got[0], got[1]) and (got[0].cpu() - want).abs().max() <= ATOL
    monkeypatch.setenv("OMNI_LORA_FOLD", "1")
    lora["lora_indices"] = torch.full((B,), 5, dtype=torch.int32, device=dev)
    with pytest.raises(IndexError):
        bad = fa.omni_attn(q.to(dev), *cache, user_id=6, n_splits=1, **lora)
        _lib.check_device_status(dev)
    assert torch.equal(bad, fa.omni_attn(q.to(dev), *cache, user_id=6, n_splits=1))


@pytest.mark.parametrize("B,H,S", [(32, 32, 300), (1, 80, 4096)])
def test_wide_costs_what_the_fp32_kernel_costs(dev, B, H, S, monkeypatch):
    """The work units go round all SMs first: with twelve consecutive units per CTA and only the heads' own CTAs, 1.4 and 2 times
    the time of the fp32 kernel launched for the call."""
    fa = attn_mod()
    gen = torch.Generator(device=dev).manual_seed(1)
    nib = torch.randint(0, 256, (B, H, S, 64), device=dev, dtype=torch.uint8, generator=gen)
    qjl = torch.randint(0, 256, (B, H, S, 8), device=dev, dtype=torch.uint8, generator=gen)
    norms = torch.rand(B, H, S, device=dev, generator=gen)
    q = torch.randn(B, H, 1, 128, device=dev, generator=gen, dtype=torch.bfloat16)
    cb = torch.linspace(-16.0, 16.0, 16, device=dev).expand(H, 16).contiguous()
    us = {}
    for kernel in ("mma", "lane"):
        monkeypatch.setenv("OMNI_QATTN_KERNEL", kernel)
        us[kernel] = device_us(lambda: fa.omni_attn(q, nib, qjl, norms, nib, cb))
    assert us["mma"] <= 1.3 * us["lane"], us          # 1.10 and 1.17 as measured
