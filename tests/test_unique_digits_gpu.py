"""sort_unique_sum where the width of its digits, the form of its scatter and the number of its chunks
and rounds change: keys against torch.unique, sums against sums in fp64 within the bound of fp32
additions in any order, (m - 1) 2^-24 sum |v| for a key of m values, and sums of whole numbers exactly.

Up to 4 718 592 ids of 16 to 42 bits (to 51 up to 786 432) are summed piece by piece, unless they crowd
together: the cases of those sizes hold that way to the same results, and the ones marked `general` make
sure that they go pass by pass."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(keys, vals, bits, general=False):
    from ps_lite_b200 import _lib
    from ps_lite_b200.ops.keys import sort_unique_sum
    want, inverse, times = torch.unique(keys, return_inverse=True, return_counts=True)
    before = _lib.device_lib().psdev_launch_count()
    got, sums = sort_unique_sum(keys, vals, key_bits=bits)
    if general:    # (pieces take three launches, buckets six)
        assert _lib.device_lib().psdev_launch_count() - before > 6
    assert torch.equal(got, want)
    exact = torch.zeros(want.numel(), dtype=torch.float64, device=keys.device)
    size = torch.zeros_like(exact)
    exact.index_add_(0, inverse, vals.double())
    size.index_add_(0, inverse, vals.double().abs())
    assert bool(((sums.double() - exact).abs() <= (times - 1) * 2.0 ** -24 * size).all())
    if general and 8 * keys.numel() < 1 << 24:
        whole = (vals * 3).round().clamp(-7, 7)
        exact.zero_().index_add_(0, inverse, whole.double())
        assert torch.equal(sort_unique_sum(keys, whole, key_bits=bits)[1].double(), exact)


# one tile of the one-CTA sort, chunks that grow until there are 32 of them, chunks of more than the
# smallest size, the larger tiles, and where keys of more than 32 bits go back to digits of 8 bits
@pytest.mark.parametrize("n", [4096, 4097, 32 * 2048, 32 * 2048 + 1, 296 * 2048 + 1, 296 * 4096,
                               296 * 4096 + 1, 1 << 21, (1 << 21) + 1])
@pytest.mark.parametrize("bits", [17, 30, 32, 33, 40])
def test_sizes(cuda_device, n, bits):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n + bits)
    keys = torch.randint(0, 1 << bits, (n,), device=cuda_device, generator=g)
    keys[::3] = keys[0]                                # a popular id
    keys[1::5] = (1 << bits) - 1 - keys[1::5] % 1000   # some hundred, at the upper end
    _check(keys, torch.randn(n, device=cuda_device, generator=g), bits)


# the chunks whose counts the scatter adds up: 16 of digits of 10 bits, 32 (of up to 4096) of 8, which
# keys of more than 40 bits have in between
@pytest.mark.parametrize("n", [16 * 2048, 16 * 2048 + 1, 29 * 2560, 80 << 10, 32 * 4096, 32 * 4096 + 1])
@pytest.mark.parametrize("bits", [8, 24, 30, 40, 48, 56, 60, 62])
def test_sizes_of_a_few_chunks(cuda_device, n, bits):
    test_sizes(cuda_device, n, bits)


# runs of equal keys that fill rounds of 2048 pairs, end with them or cross many of them
@pytest.mark.parametrize("bits", [30, 40, 52, 56])
@pytest.mark.parametrize("run", [1, 2047, 2048, 2049, 40 * 2048, 200_000])
def test_runs(cuda_device, run, bits):
    n = 200_000
    keys = torch.arange(n, device=cuda_device) // run * 4099
    g = torch.Generator(device=cuda_device)
    g.manual_seed(run)
    order = torch.randperm(n, device=cuda_device, generator=g)
    _check(keys[order], torch.randn(n, device=cuda_device, generator=g), bits, general=bits > 51)


@pytest.mark.parametrize("bits", [8, 15])
@pytest.mark.parametrize("run", [2047, 2048, 2049, 40 * 2048, 200_000])
def test_runs_of_few_bits(cuda_device, run, bits):
    n = 200_000
    g = torch.Generator(device=cuda_device)
    g.manual_seed(run)
    order = torch.randperm(n, device=cuda_device, generator=g)
    keys = torch.arange(n, device=cuda_device) // run * (1 if bits == 8 else 331)
    assert int(keys.max()) < 1 << bits
    _check(keys[order], torch.randn(n, device=cuda_device, generator=g), bits, general=bits > 8)


# one run over so many rounds of 2048 pairs: what a warp looks at first, then 512 at a time, and the
# 2048 rounds whose counts are put together at a time
ROUNDS = [31, 32, 33, 34, 543, 544, 545, 546, 1057, 2047, 2048, 2049, 4100]


def _run_over_rounds(dev, rounds, low, middle, high, others=0):
    """A run of `middle` in between 3000 smaller keys and 5000 larger ones, or `others` more of each."""
    g = torch.Generator(device=dev)
    g.manual_seed(rounds)
    first, last = 3000 + others, 5000 + others    # (smaller ones, so that the run begins inside a round)
    keys = torch.full((first + rounds * 2048 + last,), middle, device=dev)
    keys[:first] = torch.randint(low, middle, (first,), device=dev, generator=g)
    keys[-last:] = torch.randint(middle + 1, high, (last,), device=dev, generator=g)
    order = torch.randperm(keys.numel(), device=dev, generator=g)
    return keys[order], torch.randn(keys.numel(), device=dev, generator=g)


@pytest.mark.parametrize("bits", [30, 40])
@pytest.mark.parametrize("rounds", ROUNDS)
def test_a_run_over_many_rounds(cuda_device, rounds, bits):
    _check(*_run_over_rounds(cuda_device, rounds, 0, 1 << 20, 1 << bits), bits)


# the same pass by pass: keys of few bits in one word with their values, of many in arrays, and crowds
# of either kind of the widths that have wide digits
@pytest.mark.parametrize("bits", [15, 52])
@pytest.mark.parametrize("rounds", ROUNDS)
def test_a_run_over_many_rounds_pass_by_pass(cuda_device, rounds, bits):
    _check(*_run_over_rounds(cuda_device, rounds, 0, 1 << (bits - 1), 1 << bits), bits, general=True)


@pytest.mark.parametrize("bits", [24, 30, 40])
@pytest.mark.parametrize("rounds", [r for r in ROUNDS if 544 < r < 2050])
def test_a_run_among_a_crowd(cuda_device, rounds, bits):
    _check(*_run_over_rounds(cuda_device, rounds, 1 << 20, 9 << 17, 5 << 18, others=200_000), bits, general=True)


# where pairs of one word become arrays of keys and values until the last pass: two to four passes of
# 8 bits, chunks of several tiles, ends inside a tile
@pytest.mark.parametrize("n", [3 << 19, (3 << 19) + 1, (3 << 19) + 4095, 2_500_000, (1 << 22) + 12_345])
@pytest.mark.parametrize("bits", [5, 8, 16, 24, 32])
def test_keys_and_values_apart(cuda_device, n, bits):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n + bits)
    keys = torch.randint(0, 1 << bits, (n,), device=cuda_device, generator=g)
    keys[::7] = (1 << bits) - 1
    _check(keys, torch.randn(n, device=cuda_device, generator=g), bits)


@pytest.mark.parametrize("n", [(3 << 19) + 1, 2_500_000])
def test_a_key_wider_than_stated_among_many(cuda_device, n):
    """The first pass, which narrows the keys, sees it: keys sort by their low bits, as in sort_keys."""
    from ps_lite_b200.ops.keys import sort_unique_sum
    keys = torch.arange(n, device=cuda_device) % 1000
    keys[n // 2] += 1 << 40
    got, sums = sort_unique_sum(keys, torch.ones(n, device=cuda_device), key_bits=24)
    assert int(sums.sum()) == n and bool(((got & 0xffffff).diff() >= 0).all())
    assert (1 << 40) + n // 2 % 1000 in got.tolist()


# more rounds than have their counts put together at a time (2048, of 2048 pairs), and the sizes from
# which 30 bits take digits of 8 bits
@pytest.mark.parametrize("n,bits", [(1 << 22, 30), ((1 << 22) + 1, 30), ((1 << 22) + 1, 40), (9_000_000, 30),
                                    (9_000_000, 40), (1 << 25, 30), ((1 << 25) + 1, 30)])
def test_many_rounds(cuda_device, n, bits):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n)
    keys = torch.randint(0, 1 << bits, (n,), device=cuda_device, generator=g)
    # ids of which the sorted list has a run around the pair that begins the 2049th round
    middle = torch.sort(keys).values[min(n - 1, 1 << 22)]
    keys[torch.randperm(n, device=cuda_device, generator=g)[:9000]] = middle
    _check(keys, torch.randn(n, device=cuda_device, generator=g), bits)
