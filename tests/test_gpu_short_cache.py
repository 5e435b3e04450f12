"""The fp32 kernel for short caches (``OMNI_QATTN_KERNEL=short`` takes it wherever it can serve the call) against the CPU
oracle: edges of its 64-key passes and of its tiles of one, two and four query columns.

Tolerance.  Both sides sum in fp32.  A score is scale * (128 products of size 0.6 on average + the sign term), about 10 in
all; 192 additions round it by at most 192 * 2^-24 * 10 = 1.1e-4, and a score error of d moves an output by at most
2 d max|centroid| < 8 d.  Errors do not line up: a tenth of that worst case is asserted, 1e-4."""
import pytest
import torch

import oracle as orc
from tests.helpers import device_us
from tests.test_gpu_attention import make_cache, to_dev, attn_mod

pytestmark = pytest.mark.gpu

ATOL = 1e-4


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    return torch.device("cuda:0")


@pytest.fixture(autouse=True)
def force_short(monkeypatch):
    monkeypatch.setenv("OMNI_QATTN_KERNEL", "short")
    yield
    from omnistack_rs_b200 import _lib
    _lib.check_device_status(torch.device("cuda:0"))


@pytest.mark.parametrize("Hq,Hkv,T", [(3, 3, 1), (4, 2, 1), (3, 1, 1), (8, 2, 1), (5, 1, 1), (2, 1, 5)])
@pytest.mark.parametrize("S", [1, 8, 63, 64, 65, 129])
def test_short_cache_matches_oracle(dev, Hq, Hkv, T, S):
    fa = attn_mod()
    kn, kq, kr, vn, cb, gen = make_cache(3, Hkv, S, seed=Hq * 1000 + S + T, user_id=2, per_head=(Hkv != 2))
    q = torch.randn(3, Hq, T, 128, generator=gen).to(torch.bfloat16 if S % 2 else torch.float32)
    d = to_dev(dev, q, kn, kq, kr, vn, cb)
    assert (fa.omni_attn(*d, user_id=2, n_splits=1).cpu() - orc.decode_attention(q, kn, kq, kr, vn, cb, 2)).abs().max() <= ATOL
    got = fa.omni_attn(*d, user_id=2, with_qjl=False, n_splits=1).cpu()
    assert (got - orc.decode_attention(q, kn, kq, kr, vn, cb, 2, None, False)).abs().max() <= ATOL
    # ragged lengths (one user with none), V in the pair layout: the same bits as from the reference layout
    lens = torch.tensor([S, 0, max(1, S - 3)], dtype=torch.int32)
    paired = d[4].clone()
    fa.pair_v_rows(paired, 0, lens.to(dev).to(torch.int64))
    ref = fa.omni_attn(*d, user_id=2, seq_lens=lens.to(dev), n_splits=1)
    pair = fa.omni_attn(*d[:4], paired, d[5], user_id=2, seq_lens=lens.to(dev), n_splits=1, v_paired=True)
    assert torch.equal(ref, pair) and not ref[1].any()
    n = int(lens[2])
    want = orc.decode_attention(q[2:], kn[2:, :, :n], kq[2:, :, :n], kr[2:, :, :n], vn[2:, :, :n], cb, 2)
    assert (ref[2:].cpu() - want).abs().max() <= ATOL


def test_short_cache_rotation_and_slots(dev):
    fa = attn_mod()
    kn, kq, kr, vn, cb, gen = make_cache(4, 2, 70, seed=11, user_id=1)
    q = torch.randn(2, 6, 1, 128, generator=gen)
    slots = torch.tensor([3, 0], dtype=torch.int32)
    got = fa.omni_attn(q.to(dev), *to_dev(dev, kn, kq, kr, vn, cb), user_id=1, cache_slots=slots.to(dev), rotate_q=True, unrotate_out=True,
                       scale=0.07, n_splits=1).cpu()
    pick = lambda x: x[slots.long()]  # noqa: E731
    want = orc.wht128(orc.decode_attention(orc.wht128(q), pick(kn), pick(kq), pick(kr), pick(vn), cb, 1, 0.07))
    assert (got - want).abs().max() <= ATOL


@pytest.mark.parametrize("Hq,Hkv,T,hid,rank", [(8, 8, 1, 128, 16), (8, 2, 1, 128, 32), (6, 2, 1, 100, 6), (4, 2, 3, 256, 40),
                                                (8, 8, 1, 128, 32), (4, 2, 1, 128, 32), (5, 1, 1, 128, 32),       # 1, 2 and 5 columns
                                                (8, 8, 1, 128, 8), (4, 2, 1, 128, 8), (5, 1, 1, 128, 8)])
def test_short_cache_query_update(dev, Hq, Hkv, T, hid, rank, monkeypatch):
    """The per-user query update inside the kernel equals the separate launch bit for bit, index -1 leaves the query alone
    and an index past the adapters is reported."""
    fa = attn_mod()
    from omnistack_rs_b200 import _lib
    B = 5
    kn, kq, kr, vn, cb, gen = make_cache(B, Hkv, 50, seed=rank, user_id=6)
    q = torch.randn(B, Hq, T, 128, generator=gen).to(torch.bfloat16)
    x = torch.randn(B, T, hid, generator=gen)
    la = torch.randn(5, rank, hid, generator=gen) * (0.5 / hid ** 0.5)
    lb = torch.randn(5, Hq * 128, rank, generator=gen) * (0.5 / rank ** 0.5)
    idx = torch.tensor([-1, 0, 4, 2, 2], dtype=torch.int32)
    cache = to_dev(dev, kn, kq, kr, vn, cb)
    lora = dict(x=x.to(dev), lora_a=la.to(dev), lora_b=lb.to(dev), lora_indices=idx.to(dev), lora_alpha=0.3)
    got = []
    for flag in ("1", "0"):
        monkeypatch.setenv("OMNI_LORA_FOLD", flag)
        got.append(fa.omni_attn(q.to(dev), *cache, user_id=6, n_splits=1, **lora))
    want = orc.decode_attention(orc.apply_lora_to_q(q, x, la, lb, idx, 0.3), kn, kq, kr, vn, cb, 6)
    assert torch.equal(got[0], got[1]) and (got[0].cpu() - want).abs().max() <= ATOL
    monkeypatch.setenv("OMNI_LORA_FOLD", "1")
    lora["lora_indices"] = torch.full((B,), 5, dtype=torch.int32, device=dev)
    with pytest.raises(IndexError):
        bad = fa.omni_attn(q.to(dev), *cache, user_id=6, n_splits=1, **lora)
        _lib.check_device_status(dev)
    assert torch.equal(bad, fa.omni_attn(q.to(dev), *cache, user_id=6, n_splits=1))


@pytest.mark.parametrize("S", [1, 17, 64, 127])
def test_more_ctas_than_four_per_sm(dev, S):
    """One column and 600 CTAs: the build for eight CTAs per SM, which the default route takes too."""
    fa = attn_mod()
    kn, kq, kr, vn, cb, gen = make_cache(75, 8, S, seed=S, user_id=3)
    q = torch.randn(75, 8, 1, 128, generator=gen).to(torch.float16)
    d = to_dev(dev, q, kn, kq, kr, vn, cb)
    lens = torch.randint(0, S + 1, (75,), generator=gen, dtype=torch.int32)
    lens[0], lens[1] = S, 0
    assert (fa.omni_attn(*d, user_id=3, n_splits=1).cpu() - orc.decode_attention(q, kn, kq, kr, vn, cb, 3)).abs().max() <= ATOL
    few = [fa.omni_attn(*[x[b:b + 25] for x in d[:5]], d[5], user_id=3, seq_lens=lens[b:b + 25].to(dev), n_splits=1) for b in (0, 25, 50)]
    many = fa.omni_attn(*d, user_id=3, seq_lens=lens.to(dev), n_splits=1)
    assert (many - torch.cat(few)).abs().max() <= 1e-5 and not many[1].any()


def test_rank_32_costs_little_more_than_rank_16(dev, monkeypatch):
    """All rows of a rank-32 update are requested ahead, as those of rank 16 (16 users x 8 heads x 50 keys: 5.5 us;
    with the general form 9.8)."""
    monkeypatch.delenv("OMNI_QATTN_KERNEL")
    fa = attn_mod()
    kn, kq, kr, vn, cb, gen = make_cache(16, 8, 50, seed=1, user_id=3)
    cache = to_dev(dev, torch.randn(16, 8, 1, 128, generator=gen).to(torch.bfloat16), kn, kq, kr, vn, cb)
    us = {}
    for rank in (16, 32):
        lora = dict(x=torch.randn(16, 1, 128, generator=gen).to(dev), lora_a=torch.randn(4, rank, 128, generator=gen).to(dev),
                    lora_b=torch.randn(4, 8 * 128, rank, generator=gen).to(dev), lora_indices=(torch.arange(16) % 4).int().to(dev))
        us[rank] = device_us(lambda: fa.omni_attn(*cache, user_id=3, n_splits=1, **lora))
    assert us[32] <= 1.35 * us[16], us
