"""The windowed boundary search of the Lloyd-Max kernel against a plain restatement of the iterations with fp64 means:
identical boundaries give identical sums, so a few iterations agree to the rounding of the means (2 fp32 ulps of the data's
scale, the kernel's prefix sums being fp64)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def lloyd_iterations(x, iters):
    x = x.float().sort().values
    per = x.numel() // 16
    c = torch.stack([x[i * per:(i + 1) * per].double().mean() for i in range(16)]).float()
    for _ in range(iters):
        level = (x[:, None] - c[None, :]).abs().argmin(dim=1)
        n = torch.bincount(level, minlength=16)
        s = torch.zeros(16, dtype=torch.float64).index_add_(0, level, x.double())
        c = torch.where(n > 0, (s / n.clamp(min=1)).float(), c)
    return c.sort().values


def samples(kind, gen):
    if kind == "sixteen":
        return torch.randn(16, generator=gen)
    if kind == "odd":
        return torch.randn(4097, generator=gen)
    if kind == "jumps":                       # boundaries move by thousands of positions in one iteration
        return torch.cat([torch.randn(9000, generator=gen) * 0.01 + k * k for k in (-3.0, 0.0, 1.0, 5.0)])
    if kind == "few_values":
        return torch.tensor([-1.0, 0.5, 0.5000001, 3.0])[torch.randint(0, 4, (5000,), generator=gen)]
    return torch.randn(30000, generator=gen) ** 3          # heavy tails


@pytest.mark.parametrize("kind", ["sixteen", "odd", "jumps", "few_values", "heavy"])
@pytest.mark.parametrize("iters", [1, 2, 7])
def test_search_matches_assignment(kind, iters):
    from omnistack_rs_b200.quantization import calibrate_per_group
    x = samples(kind, torch.Generator().manual_seed(len(kind)))
    other = torch.randn(1000, generator=torch.Generator().manual_seed(1))
    got = calibrate_per_group([other.cuda(), x.cuda()], max_iters=iters).cpu()[1]
    assert (got - lloyd_iterations(x, iters)).abs().max() <= 2 * 2.0 ** -23 * float(x.abs().max())


@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
@pytest.mark.parametrize("first", [False, True])
def test_groups_beside_one_that_is_not_finite(bad, first):
    """A group with an infinite or NaN sample has no finite codebook; the other groups of the call get theirs as without it."""
    from omnistack_rs_b200.quantization import calibrate_per_group
    gen = torch.Generator().manual_seed(3)
    groups = [torch.randn(n, generator=gen).cuda() for n in (5000, 300, 70000)]
    spoilt = torch.randn(4000, generator=gen).cuda()
    spoilt[17] = bad
    alone = calibrate_per_group(groups, max_iters=40)
    both = calibrate_per_group([spoilt] + groups if first else groups + [spoilt], max_iters=40)
    assert not both[0 if first else 3].isfinite().all()
    rest = both[1:] if first else both[:3]
    # behind other samples the prefix sums of a group start at another value: their fp64 rounding, 2^-53 * 1e5 samples * 3, is far
    # below an fp32 ulp of a mean, which it can still move across a rounding boundary, and the iterations carry that on
    assert torch.equal(rest, alone) if not first else (rest - alone).abs().max() <= 1e-5
