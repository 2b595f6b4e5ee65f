"""One-rank keyed requests in one pass (psdev_sparse_local) against the three kernels that several
ranks use (scatter, apply, respond) on a second table: the arithmetic per value is the same, so
answers and state agree bit for bit, except where a key is repeated (its gradients are then added
in another order)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SPACE = 1 << 16


def _pair(dev, max_keys, **kw):
    from ps_lite_b200.parallel import SparseTable, SymmetricHeap
    out = []
    for _ in range(2):
        heap = SymmetricHeap((8 << 20) + max_keys * kw.get("width", 1) * 64 + 8 * SPACE *
                             kw.get("width", 1), 0, 1, device=dev)
        out.append(SparseTable(heap, SPACE, max_keys, alpha=0.1, beta=1.0, l1=0.1, l2=1.0, lr=0.3,
                               **kw))
    return out


def _three(t, keys, vals, lens=None):
    t.stage(keys, vals, lens)
    t.scatter()
    t.apply()
    t.respond()
    return t.out[: t.count_vals]


def _same_state(a, b):
    assert torch.equal(a.w, b.w)
    if a.kind == "ftrl":
        assert torch.equal(a.z, b.z) and torch.equal(a.n, b.n)


@pytest.mark.parametrize("n", [1, 2, 255, 1023, 1024, 1025, 20_000])
@pytest.mark.parametrize("kind", ["sum", "sgd", "ftrl"])
@pytest.mark.parametrize("width", [1, 3, 4, 16])
@pytest.mark.parametrize("store", ["direct", "hash"])
def test_fixed_width(cuda_device, n, kind, width, store):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n * width)
    # (room for every key there is: which key finds a full table depends on the order of arrival)
    kw = {"hash_capacity": 1 << 17} if store == "hash" else {}
    a, b = _pair(cuda_device, n, kind=kind, width=width, **kw)
    for step in range(3):
        keys = torch.sort(torch.randperm(SPACE, device=cuda_device, generator=g)[:n]).values
        if store == "direct":
            keys[-1] = SPACE + 5 if step == 1 else keys[-1]     # beyond the range: dropped
        vals = torch.randn(n * width, device=cuda_device, generator=g)
        vals[::7] = 0.0                                          # a zero changes nothing
        a.out.fill_(7.0), b.out.fill_(7.0)
        # (an odd place for the request's values: no 16-byte accesses)
        shift = step % 2
        mine = torch.cat([vals.new_zeros(shift), vals])[shift:]
        assert torch.equal(a.push_pull(keys, mine), _three(b, keys, vals))
        if store == "direct":
            _same_state(a, b)
    # pull alone, of known and unknown keys
    ask = torch.sort(torch.randperm(SPACE, device=cuda_device, generator=g)[:n]).values
    assert torch.equal(a.pull(ask), _three(b, ask, torch.zeros(n * width, device=cuda_device)))


@pytest.mark.parametrize("kind, width", [("ftrl", 1), ("sgd", 1), ("sgd", 4), ("ftrl", 3),
                                         ("sgd", 31), ("sgd", 32)])
@pytest.mark.parametrize("more", [-1, 0])
def test_one_key_per_line(cuda_device, kind, width, more):
    """Either side of the number of keys from which lines are read whole."""
    g = torch.Generator(device=cuda_device)
    g.manual_seed(width)
    value = 4 * width * (4 if kind == "ftrl" else 1)
    n = SPACE // max(1, 128 // value) + more
    a, b = _pair(cuda_device, n, kind=kind, width=width)
    for _ in range(2):
        keys = torch.sort(torch.randperm(SPACE, device=cuda_device, generator=g)[:n]).values
        vals = torch.randn(n * width, device=cuda_device, generator=g)
        assert torch.equal(a.push_pull(keys, vals), _three(b, keys, vals))
        _same_state(a, b)


@pytest.mark.parametrize("width", [1, 4, 5])
def test_repeated_keys(cuda_device, width):
    a, b = _pair(cuda_device, 4000, kind="sgd", width=width)
    keys = torch.arange(4000, device=cuda_device) // 3 * 11
    vals = torch.randn(4000 * width, device=cuda_device)
    x, y = a.push_pull(keys, vals), _three(b, keys, vals)
    # three additions in another order: a unit in the last place of values below 8
    torch.testing.assert_close(x, y, rtol=0, atol=2e-6)
    assert torch.equal(x.view(-1, width)[0:3998:3], x.view(-1, width)[1:3999:3])


@pytest.mark.parametrize("n", [1, 127, 128, 129, 8192, 8193, 40_000])
@pytest.mark.parametrize("kind", ["sum", "ftrl"])
@pytest.mark.parametrize("width", [1, 5, 8])
def test_values_with_lengths(cuda_device, n, kind, width):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n + width)
    a, b = _pair(cuda_device, n, kind=kind, width=width, var_len=True)
    keys = torch.sort(torch.randperm(SPACE, device=cuda_device, generator=g)[:n]).values
    lens = torch.randint(0, width + 1, (n,), device=cuda_device, generator=g, dtype=torch.int32)
    vals = torch.randn(int(lens.sum()), device=cuda_device, generator=g)
    for _ in range(2):
        assert torch.equal(a.push_pull(keys, vals, lens), _three(b, keys, vals, lens))
        _same_state(a, b)
        assert torch.equal(a.klen, b.klen)
    ask = torch.sort(torch.randperm(SPACE, device=cuda_device, generator=g)[:n]).values
    got, got_lens = a.pull(ask)
    want_lens = b.klen[ask]
    assert torch.equal(got_lens, want_lens)
    rows = b.w.contiguous().view(-1, width)
    mask = torch.arange(width, device=cuda_device)[None] < want_lens[:, None]
    assert torch.equal(got, rows[ask][mask])


@pytest.mark.parametrize("n", [300_000])
def test_lengths_over_several_blocks_per_chunk(cuda_device, n):
    """More keys than 2048 blocks of 128: a CTA walks several blocks."""
    from ps_lite_b200.parallel import SparseTable, SymmetricHeap
    space, width = 1 << 20, 3
    t = SparseTable(SymmetricHeap(64 << 20, 0, 1, device=cuda_device), space, n, kind="sum",
                    width=width, var_len=True)
    keys = torch.sort(torch.randperm(space, device=cuda_device)[:n]).values
    lens = (keys % (width + 1)).int()
    vals = torch.randn(int(lens.sum()), device=cuda_device)
    assert torch.equal(t.push_pull(keys, vals, lens), vals)
    got, got_lens = t.pull(keys)
    assert torch.equal(got, vals) and torch.equal(got_lens, lens)
