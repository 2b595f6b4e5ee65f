"""sort_unique_sum where the host does not hear of the sample in time, and from several threads."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

# pieces of the input whose crowds the host decides about, buckets of either kind of key
CALLS = [(700_000, 30), (700_000, 40), (1 << 20, 30), (1 << 20, 40)]


def _keys(kind, n, bits, dev, seed=0):
    g = torch.Generator(device=dev)
    g.manual_seed(n + bits + seed)
    keys = torch.randint(0, 1 << bits, (n,), device=dev, generator=g)
    if kind == "crowded":
        keys %= 1 << 15
    return keys, torch.randint(-3, 4, (n,), device=dev, generator=g).float()


def _check(keys, vals, got, sums):
    want, inverse = torch.unique(keys, return_inverse=True)
    exact = torch.zeros(want.numel(), dtype=torch.int64, device=keys.device)
    exact.index_add_(0, inverse, vals.long())
    assert torch.equal(got, want) and torch.equal(sums.long(), exact)


@pytest.mark.parametrize("kind", ["spread", "crowded"])
@pytest.mark.parametrize("n,bits", CALLS)
def test_behind_a_busy_stream(cuda_device, n, bits, kind):
    """The sample cannot be looked at for 30 ms: the host goes on without it, within a fraction of a
    millisecond, and the kernels decide."""
    from ps_lite_b200 import _lib
    from ps_lite_b200.ops.keys import sort_unique_sum
    count = _lib.device_lib().psdev_launch_count
    keys, vals = _keys(kind, n, bits, cuda_device)
    sort_unique_sum(keys, vals, key_bits=bits)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream(cuda_device)
    # launches before the host looks for the sample, and with those of the pieces or buckets
    some, most = (1, 2) if n < 1 << 20 else (2, 5)

    def call(out):
        torch.cuda.set_device(cuda_device)
        with torch.cuda.stream(stream):
            torch.cuda._sleep(60_000_000)          # (clocks: some 30 ms)
            out.append(sort_unique_sum(keys, vals, key_bits=bits))

    def gap():
        before, begun, done, out = count(), None, None, []
        t = threading.Thread(target=call, args=(out,))
        t.start()
        until = time.perf_counter() + 2
        while done is None and time.perf_counter() < until:
            have = count() - before
            if begun is None and have >= some:
                begun = time.perf_counter()
            if have >= most:
                done = time.perf_counter()
        busy = not stream.query()
        t.join()
        stream.synchronize()
        _check(keys, vals, *out[0])
        assert busy
        return done - begun
    assert min(gap() for _ in range(3)) < 0.6e-3   # (of three: the test's thread may be held up)


def test_calls_of_several_threads(cuda_device):
    """Each on a stream of its own, of all routes, crowded and spread keys in turn."""
    from ps_lite_b200.ops.keys import sort_unique_sum
    sets = [_keys(kind, n, bits, cuda_device, s) for s, (n, bits) in
            enumerate(CALLS + [(5000, 30), (100_000, 40), (300_000, 30), (1_000_000, 56)])
            for kind in ("spread", "crowded")]
    widths = [b for _, b in CALLS + [(5000, 30), (100_000, 40), (300_000, 30), (1_000_000, 56)] for _ in "12"]
    torch.cuda.synchronize()
    bad = []

    def run(first):
        try:
            torch.cuda.set_device(cuda_device)
            with torch.cuda.stream(torch.cuda.Stream(cuda_device)):
                for i in range(24):
                    j = (first + i) % len(sets)
                    got = sort_unique_sum(*sets[j], key_bits=widths[j])
                    torch.cuda.current_stream().synchronize()
                    _check(*sets[j], *got)
        except BaseException as e:  # noqa: BLE001
            bad.append((first, repr(e)))
    threads = [threading.Thread(target=run, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad
