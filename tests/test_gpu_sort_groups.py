"""``omni_sort_groups`` against torch's sort, group by group: sizes at the edges of a 4,096-sample chunk, repeated values, signed
zeros, infinities and NaN (last, whatever its sign)."""
import itertools

import pytest
import torch

from omnistack_rs_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [4095, 4096, 4097], [16, 100000, 1, 33], [300, 0x12345, 7]])
def test_sort_groups_matches_torch(sizes):
    dev = torch.device("cuda:0")
    lib = _lib.ensure_init(dev)
    gen = torch.Generator().manual_seed(sum(sizes))
    groups = [torch.randn(n, generator=gen) * 10.0 ** float(torch.randint(-30, 30, (1,), generator=gen)) for n in sizes]
    big = max(groups, key=len)
    if big.numel() > 30:
        big[::3] = big[0]
        big[1:9] = torch.tensor([float("nan"), -float("nan"), float("inf"), -float("inf"), 0.0, -0.0, 1e-42, -1e-42])
    flat = torch.cat(groups).to(dev)
    chunks = [-(-n // 4096) for n in sizes]
    off = torch.tensor(list(itertools.accumulate(sizes, initial=0)), device=dev)
    cbase = torch.tensor(list(itertools.accumulate(chunks, initial=0)), device=dev)
    nbytes = lib.omni_sort_groups_workspace_bytes(flat.numel(), len(sizes), sum(chunks))
    ws = torch.empty(nbytes // 8 + 1, dtype=torch.float64, device=dev)
    out = torch.empty_like(flat)
    _lib.check(lib.omni_sort_groups(_lib.ptr(flat), flat.numel(), _lib.ptr(off), _lib.ptr(cbase), len(sizes), sum(chunks), _lib.ptr(ws), nbytes,
                                    _lib.ptr(out), _lib.stream_ptr(dev)))
    for got, g in zip(out.cpu().split(sizes), groups):
        want = g.sort().values
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(0.0), want.nan_to_num(0.0))
    assert lib.omni_sort_groups(_lib.ptr(flat), flat.numel(), _lib.ptr(off), _lib.ptr(cbase), len(sizes), sum(chunks), _lib.ptr(ws), nbytes - 1,
                                _lib.ptr(out), None) == _lib.ERR_ARG
