"""sort_unique_sum (sort, count and segmented-sum kernels) against torch.unique and sums in fp64, at
the edges of a tile, of the one-launch form and of the chunks, for short and for 64-bit keys."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 4095, 4096, 4097, 8193, 600_001, 2_500_000])
@pytest.mark.parametrize("bits,kind", [(8, "uniform"), (30, "uniform"), (32, "uniform"),
                                       (33, "uniform"), (64, "uniform"), (30, "one"), (41, "one"),
                                       (24, "runs"), (30, "popular")])
def test_sums_of_equal_keys(cuda_device, n, bits, kind):
    from ps_lite_b200.ops.keys import sort_unique_sum
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n + bits)
    top = min(bits, 62)
    if kind == "uniform":
        keys = torch.randint(0, 1 << top, (n,), device=cuda_device, dtype=torch.int64, generator=g)
    elif kind == "one":      # a single key over all chunks
        keys = torch.full((n,), (1 << bits) - 1, device=cuda_device, dtype=torch.int64)
    elif kind == "runs":     # keys that cross every boundary of a thread, a warp, a tile
        keys = torch.arange(n, device=cuda_device, dtype=torch.int64) // 37
    else:
        keys = torch.randint(0, 1 << top, (n,), device=cuda_device, dtype=torch.int64, generator=g)
        keys[torch.rand(n, device=cuda_device, generator=g) < 0.3] = 12345
    vals = torch.randn(n, device=cuda_device, generator=g)
    before = keys.clone(), vals.clone()
    uk, sums = sort_unique_sum(keys, vals, key_bits=bits)
    assert torch.equal(keys, before[0]) and torch.equal(vals, before[1])
    ref, inv, count = torch.unique(keys, return_inverse=True, return_counts=True)
    assert torch.equal(uk, ref)
    exact = torch.zeros(ref.numel(), device=cuda_device, dtype=torch.float64)
    exact.index_add_(0, inv, vals.double())
    size = torch.zeros_like(exact).index_add_(0, inv, vals.double().abs())
    # m additions in any order: off by at most (m - 1) half units of the sum of magnitudes
    bound = (count - 1).double() * 2.0 ** -24 * size * 1.01
    assert torch.all((sums.double() - exact).abs() <= bound)


def test_keys_beyond_the_stated_width(cuda_device):
    """Keys with more bits than stated sort by their low bits, as sort_keys does."""
    from ps_lite_b200.ops.keys import sort_unique_sum
    keys = torch.tensor([5 + 256, 3, 5 + 256, 4 + 512], device=cuda_device)
    uk, sums = sort_unique_sum(keys, torch.ones(4, device=cuda_device), key_bits=8)
    assert uk.tolist() == [3, 4 + 512, 5 + 256] and sums.tolist() == [1.0, 1.0, 2.0]
