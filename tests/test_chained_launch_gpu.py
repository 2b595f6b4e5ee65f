"""Kernels launched while their predecessor still runs read what it wrote: long chains on one stream
without a wait in between, at sizes of one CTA and of several waves, against torch in the same order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4096, 3_000_064])
def test_packed_gradients_of_the_step_before(cuda_device, n):
    """Each step packs the weights that the step before published."""
    from ps_lite_b200.parallel import DenseTable, ServerOptimizer, SymmetricHeap
    heap = SymmetricHeap((1 << 20) + 6 * n, 0, 1, device=cuda_device)
    table = DenseTable(heap, n, torch.int8, torch.float32,
                       optimizer=ServerOptimizer("sgd", lr=0.25))
    torch.manual_seed(n)
    w0 = torch.randn(n, device=cuda_device)
    table.load_master(w0)
    grad = w0.clone()
    for _ in range(12):
        table.stage_int8(grad)
        table.push_pull()
        grad = table.weight  # (the arena itself: nothing lies between the two kernels)
    got = table.weight.clone()
    w, g = w0.clone(), w0.clone()
    for _ in range(12):
        x = torch.zeros((n + 255) // 256 * 256, device=cuda_device)
        x[:n] = g
        groups = x.view(-1, 256)
        top = groups.abs().amax(1, keepdim=True)
        scale = torch.where(top > 0, top / 127, torch.ones_like(top))
        q = (groups * (1 / scale)).clamp(-127, 127).round() * scale
        w = w - 0.25 * q.view(-1)[:n]
        g = w
    # a value beside a rounding boundary may take the neighbouring code: a step of the largest
    # value of its group / 127, times the learning rate, in each of the twelve steps
    step = 0.25 * w0.abs().max() / 127
    assert torch.all((got - w).abs() <= 12 * step)
    assert (got - w).abs().mean() <= 0.05 * step
    heap.close()


@pytest.mark.parametrize("n,bits", [(300, 20), (100_000, 24), (700_001, 40)])
def test_keys_written_just_before(cuda_device, n, bits):
    from ps_lite_b200.ops.keys import sort_unique_sum
    torch.manual_seed(n)
    ids = torch.randint(0, 1 << bits, (n,), device=cuda_device)
    ones = torch.ones(n, device=cuda_device)
    for step in range(6):
        ids = (ids * 5 + step) % (1 << bits)
        keys, sums = sort_unique_sum(ids, ones, key_bits=bits)
        want, counts = torch.unique(ids, return_counts=True)
        assert torch.equal(keys, want) and torch.equal(sums.long(), counts)


def test_counts_reach_the_host_from_many_threads(cuda_device):
    """More concurrent calls than there are report words in the shared page."""
    import threading

    from ps_lite_b200.ops.keys import sort_unique_sum
    ids = [torch.randint(0, 1 << 16, (3000 + 97 * i,), device=cuda_device) for i in range(72)]
    want = [torch.unique(k) for k in ids]
    got = [None] * len(ids)
    torch.cuda.synchronize()
    start = threading.Barrier(len(ids))

    def run(i):
        with torch.cuda.stream(torch.cuda.Stream(cuda_device)):
            start.wait()
            got[i] = sort_unique_sum(ids[i], torch.ones(ids[i].numel(), device=cuda_device),
                                     key_bits=16)[0]
            torch.cuda.current_stream(cuda_device).synchronize()
    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(ids))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for g, w in zip(got, want):
        assert torch.equal(g, w)


def test_keys_wider_than_said_take_the_general_form(cuda_device):
    from ps_lite_b200.ops.keys import sort_unique_sum
    for n in (1000, 50_000):
        ids = torch.arange(n, device=cuda_device) + (1 << 20)
        keys, sums = sort_unique_sum(ids, torch.ones(n, device=cuda_device), key_bits=16)
        assert keys.numel() == n and bool((sums == 1).all())
