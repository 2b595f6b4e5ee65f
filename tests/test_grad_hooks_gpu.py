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
