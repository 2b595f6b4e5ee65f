"""Several slices of a table in one launch on one rank: slices that start and end anywhere, several
of them inside the eight values that a thread takes at a time, and gaps between them."""
import pytest
import torch

from ps_lite_b200.utils.oracle import dense_update

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("multiple", [4, 1])
@pytest.mark.parametrize("kind", ["sum", "adam"])
@pytest.mark.parametrize("gdt,odt", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32),
                                     (torch.float32, torch.bfloat16), (torch.int8, torch.float32)])
def test_every_value_of_the_slices_once(cuda_device, gdt, odt, kind, multiple):
    from ps_lite_b200 import _lib
    from ps_lite_b200.parallel import DenseTable, ServerOptimizer, SymmetricHeap
    torch.manual_seed(13)
    n = 20_224   # (no padding for any type)
    heap = SymmetricHeap(4 << 20, 0, 1, device=cuda_device)
    t = DenseTable(heap, n, gdt, odt, optimizer=ServerOptimizer(kind, lr=0.01, eps=1e-6))
    w0 = torch.randn(t.n, device=cuda_device)
    t.load_master(w0)
    if gdt == torch.int8:
        t.stage_int8(torch.randn(t.n, device=cuda_device))
        grad = t.grad.float() * t.gscale.repeat_interleave(256)
    else:
        t.grad.copy_(torch.randn(t.n, device=cuda_device))
        grad = t.grad.float()
    near = [multiple * i for i in range(12)] + [1020, 1024, 1028, t.n - 4]
    cuts = sorted({0, t.n, *near, *(x - x % multiple for x in torch.randint(0, n, (60,)).tolist())})
    segs = [(b, e, (i * 7) % 13) for i, (b, e) in enumerate(zip(cuts[:-1], cuts[1:])) if i % 5 != 3]
    inside = torch.zeros(t.n, dtype=torch.bool, device=cuda_device)
    for b, e, _ in segs:
        inside[b:e] = True
    before = t.weight.clone()
    t.step = 1
    t.run_multi(_lib.OP_PUSHPULL, segs)
    new = dense_update(w0.clone(), [grad], kind, lr=0.01, eps=1e-6, step=1,
                       s1=torch.zeros_like(w0), s2=torch.zeros_like(w0))
    # a few fp32 operations per value; a bf16 weight is rounded once more
    tol = dict(rtol=2e-5, atol=2e-5) if odt == torch.float32 else dict(rtol=1e-2, atol=1e-2)
    torch.testing.assert_close(t.master, torch.where(inside, new, w0), rtol=2e-5, atol=2e-5)
    torch.testing.assert_close(t.weight[inside].float(), new[inside], **tol)
    assert torch.equal(t.weight[~inside], before[~inside])
    t.weight.zero_()
    t.run_multi(_lib.OP_PULL, segs)
    expected = torch.where(inside, t.master, torch.zeros_like(w0)).to(odt)
    assert torch.equal(t.weight, expected)
    t.check()
    heap.close()
