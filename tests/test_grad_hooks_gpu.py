"""Native gradient hooks of DistributedOptimizer on one rank: gradients of every layout, parameters
of one value up to several tiles, launches of one and of many pieces, hooks of the program beside
them, against the same SGD update in fp32 PyTorch on gradients rounded to the table's type."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch_bytes", [1, 4096, 1 << 22])
@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("wdt,gdt", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16),
                                     (torch.float32, torch.float32)])
def test_update_matches_fp32_sgd(cuda_device, batch_bytes, overlap, wdt, gdt):
    from ps_lite_b200.parallel import ServerOptimizer, SymmetricHeap
    from ps_lite_b200.parallel.optimizer import DistributedOptimizer
    torch.manual_seed(5)
    shapes = [(1,), (7,), (8,), (33, 3), (16, 4, 3, 3), (1025,), (300, 17)] + [(65,)] * 70
    params = [torch.nn.Parameter(torch.randn(s, device=cuda_device).to(wdt)) for s in shapes]
    master = [p.detach().float().clone() for p in params]
    seen = []
    heap = SymmetricHeap(4 << 20, 0, 1, device=cuda_device)
    dopt = DistributedOptimizer(params, heap, ServerOptimizer("sgd", lr=0.125), grad_dtype=gdt,
                                overlap=overlap, batch_bytes=batch_bytes)
    assert dopt._native is not None
    params[3].register_post_accumulate_grad_hook(lambda p: seen.append(tuple(p.grad.shape)))
    for _ in range(3):
        coef = [torch.randn(s, device=cuda_device).to(wdt) for s in shapes]
        # a gradient that is not contiguous: through the table's buffer
        coef[4] = coef[4].contiguous(memory_format=torch.channels_last)
        dopt.zero_grad()
        sum((p * c).sum() for p, c in zip(params, coef)).backward()
        assert all(p.grad is None for p in params)
        dopt.step()
        for m, c in zip(master, coef):
            m -= 0.125 * c.to(gdt).float()
        for p, m in zip(params, master):
            # one fused multiply-add per value: equal up to the rounding of the product
            tol = dict(rtol=1e-2, atol=1e-2) if wdt == torch.bfloat16 else dict(rtol=1e-6, atol=1e-6)
            torch.testing.assert_close(p.detach().float(), m, **tol)
    assert seen == [(33, 3)] * 3
    assert dopt.launches >= (3 if batch_bytes > 4096 else 6) and dopt.launched_slices == 3 * len(shapes)
    dopt.close()
    # the hooks are gone: gradients stay with the parameters again
    sum((p.float() ** 2).sum() for p in params).backward()
    assert all(p.grad is not None for p in params)
    heap.close()


def _ready(dopt, grads):
    """A backward pass that hands over ready gradients."""
    class Backward(torch.autograd.Function):
        @staticmethod
        def forward(ctx, *params):
            return params[0].new_zeros(())

        @staticmethod
        def backward(ctx, _):
            return tuple(grads)

    Backward.apply(*dopt.params).backward()


# launches of twelve gradients of 4 MiB: a named batch grows up to fourfold while the launch before is
# still running, the default up to 16 MiB, and an eighth of a second of other work is running
@pytest.mark.parametrize("named,launches", [(4 << 20, 4), (8 << 20, 3), (16 << 20, 2), (None, 4)])
def test_launches_wait_while_the_gpu_is_busy(cuda_device, named, launches):
    from ps_lite_b200.parallel import ServerOptimizer, SymmetricHeap
    from ps_lite_b200.parallel.optimizer import DistributedOptimizer
    n = 1 << 21
    params = [torch.nn.Parameter(torch.zeros(n, device=cuda_device, dtype=torch.bfloat16)) for _ in range(12)]
    heap = SymmetricHeap(12 * n * 8, 0, 1, device=cuda_device)
    dopt = DistributedOptimizer(params, heap, ServerOptimizer("sgd", lr=1.0), batch_bytes=named)
    assert dopt.batch_bytes == (named or 12 << 20)
    for _ in range(2):
        before = dopt.launches
        grads = [torch.ones_like(p) for p in params]
        torch.cuda.synchronize()
        torch.cuda._sleep(1 << 28)
        _ready(dopt, grads)
        dopt.step()
        torch.cuda.synchronize()
        assert dopt.launches - before == launches
    assert all(bool((p == -2.0).all()) for p in params)
    dopt.close()
    heap.close()


@pytest.mark.parametrize("mib,batch", [(8, 4), (16, 4), (24, 6), (64, 16), (160, 32)])
def test_most_gradients_go_out_before_the_step(cuda_device, mib, batch):
    """Whatever the size of the model: at most a quarter of them waits for the step."""
    from ps_lite_b200.parallel import ServerOptimizer, SymmetricHeap
    from ps_lite_b200.parallel.optimizer import DistributedOptimizer
    n = 1 << 20
    params = [torch.nn.Parameter(torch.zeros(n, device=cuda_device, dtype=torch.bfloat16))
              for _ in range(mib // 2)]
    heap = SymmetricHeap(len(params) * n * 8, 0, 1, device=cuda_device)
    dopt = DistributedOptimizer(params, heap, ServerOptimizer("sgd", lr=1.0), overlap=False)
    assert dopt.batch_bytes == batch << 20
    _ready(dopt, [torch.ones_like(p) for p in params])
    assert dopt._native.launches == mib // batch  # (without overlap nothing is held back)
    dopt.step()
    torch.cuda.synchronize()
    assert all(bool((p == -1.0).all()) for p in params)
    dopt.close()
    heap.close()
