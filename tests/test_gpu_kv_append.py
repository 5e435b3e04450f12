"""``QuantizedKVCache.append`` as one library call against the codec calls it stands for: packed bytes, pair layout, lengths,
and the errors of an append that does not fit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pair_v,residual,per_head,T,dtype", [(False, True, True, 1, torch.bfloat16), (True, True, False, 5, torch.float32),
                                                              (True, False, True, 17, torch.float16), (False, False, True, 8, torch.bfloat16)])
def test_append_equals_separate_calls(pair_v, residual, per_head, T, dtype, monkeypatch):
    from omnistack_rs_b200.serving import QuantizedKVCache
    dev = torch.device("cuda:0")
    gen = torch.Generator(device=dev).manual_seed(T)
    cb = torch.sort(torch.randn(3, 16, generator=gen, device=dev), dim=1).values
    make = lambda: QuantizedKVCache(5, 3, 64, cb if per_head else cb[0], dev, store_v_residual=residual, pair_v=pair_v)  # noqa: E731
    a, b = make(), make()
    monkeypatch.setattr(b, "_append_together", lambda *args: False)
    start = torch.tensor([0, 3, 8, 13, 64 - 2 * T], device=dev)
    for cache in (a, b):
        cache.lens.copy_(start)
        cache.lens32.copy_(start)
    for step in range(2):
        wide = torch.randn(5, T, 3, 256, generator=gen, device=dev).to(dtype)
        k, v = wide[..., :128].transpose(1, 2), wide[..., 128:].transpose(1, 2)           # strided views, read in place
        for cache in (a, b):
            cache.append(k, v)
    assert torch.equal(a.lens, start + 2 * T) and torch.equal(a.lens32.long(), a.lens)
    for name in ("k_nib", "k_qjl", "k_norms", "v_nib", "v_qjl", "v_norms", "lens", "lens32"):
        x, y = getattr(a, name), getattr(b, name)
        assert (x is None and y is None) or torch.equal(x, y), name
    before = [t.clone() for t in (a.k_nib, a.v_nib, a.lens)]
    with pytest.raises(ValueError, match="capacity"):
        a.append(k, v)                                                                    # one user is full
    a.lens[0] = -1
    a.lens[4] = 0
    with pytest.raises(ValueError, match="capacity"):
        a.append(k, v)
    assert torch.equal(a.k_nib, before[0]) and torch.equal(a.v_nib, before[1])


def test_index_range():
    from omnistack_rs_b200 import _lib
    dev = torch.device("cuda:0")
    for n in (1, 31, 33, 257, 5000):
        x = torch.randint(-10 ** 12, 10 ** 12, (n,), device=dev, generator=torch.Generator(device=dev).manual_seed(n))
        assert _lib.index_range(x) == (int(x.min()), int(x.max()))
        assert _lib.index_range(x.to(torch.int32)) == (int(x.to(torch.int32).min()), int(x.to(torch.int32).max()))
    assert _lib.index_range(torch.tensor([3, -4])) == (-4, 3)
