"""sort_unique_sum piece by piece, where its way and its parts change: keys against torch.unique, sums
against sums in fp64 within the bound of fp32 additions in any order, (m - 1) 2^-24 sum |v| for a key of
m values, which says little where m is large: there, and wherever a key's values are added up apart from
the others, sums of whole numbers, which have to be exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu

FEW, MOST = 3 << 18, 9 << 19   # items that are not scattered, items that go into buckets


def _check(keys, vals, bits):
    from ps_lite_b200.ops.keys import sort_unique_sum
    want, inverse, times = torch.unique(keys, return_inverse=True, return_counts=True)
    got, sums = sort_unique_sum(keys, vals, key_bits=bits)
    assert torch.equal(got, want)
    exact = torch.zeros(want.numel(), dtype=torch.float64, device=keys.device)
    size = torch.zeros_like(exact)
    exact.index_add_(0, inverse, vals.double())
    size.index_add_(0, inverse, vals.double().abs())
    assert bool(((sums.double() - exact).abs() <= (times - 1) * 2.0 ** -24 * size).all())
    again, same = sort_unique_sum(keys, vals, key_bits=bits)
    assert torch.equal(again, got) and torch.equal(same, sums)


def _check_exact(keys, bits):
    """Whole numbers of which every partial sum is below 2^24: any order of additions is exact."""
    from ps_lite_b200.ops.keys import sort_unique_sum
    g = torch.Generator(device=keys.device)
    g.manual_seed(keys.numel())
    vals = torch.randint(-3, 5, keys.shape, device=keys.device, generator=g)
    want, inverse = torch.unique(keys, return_inverse=True)
    exact = torch.zeros_like(want).index_add_(0, inverse, vals)
    size = torch.zeros_like(want).index_add_(0, inverse, vals.abs())
    assert int(size.max()) < 1 << 24
    got, sums = sort_unique_sum(keys, vals.float(), key_bits=bits)
    assert torch.equal(got, want) and torch.equal(sums, exact.float())


def _keys(kind, n, bits, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(n + bits)
    keys = torch.randint(0, 1 << bits, (n,), device=dev, generator=g)
    if kind == "popular":        # half of all items one id, a tenth another one
        order = torch.randperm(n, device=dev, generator=g)
        keys[order[: n // 2]] = (1 << bits) - 1
        keys[order[n // 2: n // 2 + n // 10]] = 5
    elif kind == "low":          # in a small range of a large space
        keys %= 1 << min(bits, 15)
    elif kind == "ranges":       # in a few narrow ranges
        wide = min(bits - 4, 20)
        keys = (keys >> (bits - 3) << (bits - 3)) + keys % (1 << wide)
    elif kind == "one":
        keys.fill_(3)
    elif kind == "rising":
        keys = torch.arange(n, device=dev) * ((1 << bits) // n) if n < 1 << bits else torch.sort(keys)[0]
    return keys, torch.randn(n, device=dev, generator=g)


@pytest.mark.parametrize("kind", ["spread", "popular", "low", "ranges", "one", "rising"])
@pytest.mark.parametrize("n", [4097, 5120, 65_537, 131_073, 300_001, FEW])
@pytest.mark.parametrize("bits", [16, 24, 32, 33, 40, 51])
def test_pieces_of_the_input(cuda_device, kind, n, bits):
    _check(*_keys(kind, n, bits, cuda_device), bits)


# the line up to which a sample makes the parts of crowded keys
@pytest.mark.parametrize("kind", ["spread", "popular", "low", "ranges"])
@pytest.mark.parametrize("n", [5 << 17, (5 << 17) + 1])
@pytest.mark.parametrize("bits", [24, 40])
def test_parts_by_a_sample(cuda_device, kind, n, bits):
    _check(*_keys(kind, n, bits, cuda_device), bits)


@pytest.mark.parametrize("kind", ["spread", "popular", "low", "ranges", "one", "rising"])
@pytest.mark.parametrize("n", [FEW + 1, 1 << 20, (1 << 20) + 1, 296 * 4096 + 1, MOST])
@pytest.mark.parametrize("bits", [16, 24, 32, 33, 42])
def test_buckets(cuda_device, kind, n, bits):
    _check(*_keys(kind, n, bits, cuda_device), bits)


@pytest.mark.parametrize("kind", ["spread", "popular", "low", "ranges", "one"])
@pytest.mark.parametrize("n", [4097, 5120, 65_537, 300_001, 5 << 17, FEW, FEW + 1, 1 << 20, (1 << 21) + 1, MOST])
@pytest.mark.parametrize("bits", [16, 30, 40])
def test_sums_of_whole_numbers(cuda_device, kind, n, bits):
    _check_exact(_keys(kind, n, bits, cuda_device)[0], bits)


# popular ids of a bucket: one that takes away more than a quarter of a piece's items (again and again),
# several that take less, and pieces that keep at most two rows
@pytest.mark.parametrize("n", [FEW + 1, (1 << 20) + 1, MOST])
@pytest.mark.parametrize("bits", [24, 40])
@pytest.mark.parametrize("shares", [[4], [4, 3, 3, 3, 3, 2], [8] * 10, [2, 1000], [1.05], [1.01, 200]])
def test_popular_ids_of_a_bucket(cuda_device, n, bits, shares):
    keys, _ = _keys("spread", n, bits, cuda_device)
    left = torch.randperm(n, device=cuda_device)[: n // 2]
    for j, share in enumerate(shares):      # every share-th of those that are left
        take = int(len(left) / share)
        keys[left[:take]] = (5 << (bits - 10)) + 3 * j
        left = left[take:]
    _check_exact(keys, bits)


# beyond what pieces and buckets are for
@pytest.mark.parametrize("n,bits", [(FEW, 52), (FEW + 1, 43), (MOST + 1, 30), (9000, 15)])
def test_the_general_way(cuda_device, n, bits):
    _check(*_keys("spread", n, bits, cuda_device), bits)


# distinct keys of a part or a bucket: as many as a CTA sorts, and one more
@pytest.mark.parametrize("n,bits", [(40_000, 30), (40_000, 40), (1 << 20, 30), (1 << 20, 40)])
@pytest.mark.parametrize("crowd", [5119, 5120, 5121, 12_000])
def test_a_crowd(cuda_device, n, bits, crowd):
    keys, vals = _keys("spread", n, bits, cuda_device)
    at = torch.randperm(n, device=cuda_device)[:crowd]
    keys[at] = (1 << (bits - 1)) + torch.arange(crowd, device=cuda_device)
    _check(keys, vals, bits)


# popular ids side by side, which every piece of the input has: more items for one part than a CTA sorts
@pytest.mark.parametrize("bits", [30, 40])
@pytest.mark.parametrize("ids,crowd", [(19, 0), (20, 0), (21, 0), (100, 0), (40, 3000), (40, 6000)])
def test_popular_neighbours(cuda_device, bits, ids, crowd):
    n = 400_000
    keys, vals = _keys("spread", n, bits, cuda_device)
    keys[::2] = (1 << (bits - 1)) + torch.arange(n // 2, device=cuda_device) % ids
    if crowd:
        keys[1:2 * crowd:2] = (1 << (bits - 1)) + 1000 + torch.arange(crowd, device=cuda_device)
    _check(keys, vals, bits)
    _check_exact(keys, bits)


# parts of the input with more items than a CTA sorts, which another CTA helps to merge: of one group
# (40 parts away), without a key in the first piece, with one, with more keys than both can sort
@pytest.mark.parametrize("n", [(1 << 19) + 1, 700_000, FEW])
@pytest.mark.parametrize("bits", [24, 30, 40])
@pytest.mark.parametrize("ids,parts,first,crowd", [(25, [7], True, 0), (40, [7, 47, 255], True, 0),
                                                   (30, [0, 40], True, 0), (25, [7], False, 0), (21, [9], None, 0),
                                                   (25, [7], True, 4500), (25, [7], True, 5200),
                                                   (120, [3], True, 2000)])
def test_parts_that_are_helped(cuda_device, n, bits, ids, parts, first, crowd):
    keys, _ = _keys("spread", n, bits, cuda_device)
    shift, size = bits - 8, (n + 255) // 256
    for j, part in enumerate(parts):
        at = torch.arange(j, n, 7, device=cuda_device)
        keys[at] = (part << shift) + 11 * (torch.arange(at.numel(), device=cuda_device) % ids)
    if first is not True:          # the first piece: nothing of the part, or one key
        keys[:size] = torch.where(keys[:size] >> shift == parts[0], 0, keys[:size])
        if first is None:
            keys[5] = (parts[0] << shift) + 22
    if crowd:
        keys[3:7 * crowd:7] = (parts[0] << shift) + 5000 + torch.arange(crowd, device=cuda_device)
    _check_exact(keys, bits)


# a part with some items more than a CTA sorts, of fewer keys: three of them are in each of 79 pieces
@pytest.mark.parametrize("bits", [30, 40])
def test_a_part_with_a_few_items_too_many(cuda_device, bits):
    from ps_lite_b200 import _lib
    n, first = 40_000, 1 << (bits - 1)
    keys, vals = _keys("spread", n, bits, cuda_device)
    keys[keys >> (bits - 7) == 64] += 1 << (bits - 2)       # (nothing else in the part)
    at = torch.arange(4997, device=cuda_device)
    keys[at * 8] = first + 3 + at
    keys[1::2] = torch.where(torch.arange(n // 2, device=cuda_device) % 10 == 0,
                             first + torch.arange(n // 2, device=cuda_device) // 10 % 3, keys[1::2])
    before = _lib.device_lib().psdev_launch_count()
    _check(keys, vals, bits)
    assert _lib.device_lib().psdev_launch_count() - before == 6   # (two calls: pieces, merge, gather)


@pytest.mark.parametrize("n", [9000, 600_000, FEW + 1])
@pytest.mark.parametrize("bits", [20, 40])
def test_a_key_wider_than_stated(cuda_device, n, bits):
    """Keys sort by their low bits then, as in sort_keys."""
    from ps_lite_b200.ops.keys import sort_unique_sum
    keys = torch.arange(n, device=cuda_device) % 1000 << (bits - 10)
    keys[n // 2] += 1 << 55
    got, sums = sort_unique_sum(keys, torch.ones(n, device=cuda_device), key_bits=bits)
    assert int(sums.sum()) == n and bool(((got & ((1 << bits) - 1)).diff() >= 0).all())


# the order in which the values of a key are added up does not depend on them: in the order of their
# bits all positive ones would come first, and partial sums would be large
@pytest.mark.parametrize("kind", ["low", "popular"])
@pytest.mark.parametrize("n", [4097, 65_537, 131_072, 131_073, FEW, 1 << 20])
@pytest.mark.parametrize("bits", [24, 32, 40])
def test_negated_values_have_negated_sums(cuda_device, kind, n, bits):
    from ps_lite_b200.ops.keys import sort_unique_sum
    keys, vals = _keys(kind, n, bits, cuda_device)
    ids, sums = sort_unique_sum(keys, vals, key_bits=bits)
    same, negated = sort_unique_sum(keys, -vals, key_bits=bits)
    assert torch.equal(ids, same) and torch.equal(sums, -negated)
