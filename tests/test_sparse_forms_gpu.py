"""SparseTable on one rank: requests whose tensors its kernel cannot read as they are."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("var_len", [False, True])
def test_negated_views_and_other_places(cuda_device, var_len):
    from ps_lite_b200.parallel import SparseTable, SymmetricHeap
    heap = SymmetricHeap(4 << 20, 0, 1, device=cuda_device)
    table = SparseTable(heap, 1 << 12, 600, kind="sum", width=4, var_len=var_len)
    keys = torch.randperm(1 << 12)[:500].sort().values.to(cuda_device)
    lens = (torch.arange(500, dtype=torch.int32) % 4 + 1).to(cuda_device) if var_len else None
    count = int(lens.sum()) if var_len else 2000
    vals = torch.randint(-9, 9, (count,), device=cuda_device).float()
    want = torch.zeros(count, device=cuda_device)
    forms = [(keys, vals, lens, 1), (keys, torch._neg_view(vals), lens, -1),
             (keys.cpu(), vals, lens, 1), (keys, vals.cpu(), lens, 1),
             (keys, vals, lens.cpu() if var_len else None, 1)]
    if torch.cuda.device_count() > 1:
        forms += [(keys.to("cuda:1"), vals.to("cuda:1"), lens.to("cuda:1") if var_len else None, 1)]
    for k, v, l, sign in forms:
        got = table.push_pull(k, v, l)
        want += sign * vals
        assert torch.equal(got, want)
        pulled = table.pull(k)
        assert torch.equal(pulled[0] if var_len else pulled, want)
    with pytest.raises(RuntimeError):
        table.push_pull(torch._neg_view(-keys), vals, lens)   # refused by torch, as ever
    heap.close()
