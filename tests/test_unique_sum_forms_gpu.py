"""sort_unique_sum: arguments that its kernels cannot take as they are go the general way, which follows
them as torch does, or stay refused."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_tangents_and_graphs(cuda_device):
    from torch.autograd import forward_ad

    from ps_lite_b200.ops.keys import sort_unique_sum
    keys = torch.tensor([5, 3, 5, 9, 3, 5], device=cuda_device)
    vals, tang = torch.arange(6.0, device=cuda_device), torch.arange(10.0, 16.0, device=cuda_device)
    want, want_t = torch.tensor([5.0, 7.0, 3.0]), torch.tensor([25.0, 37.0, 13.0])
    with forward_ad.dual_level():
        uk, sums = sort_unique_sum(keys, forward_ad.make_dual(vals, tang), key_bits=8)
        value, tangent = forward_ad.unpack_dual(sums)
        assert uk.tolist() == [3, 5, 9] and torch.equal(value.cpu(), want)
        assert tangent is not None and torch.equal(tangent.cpu(), want_t)
    # inside a transform of torch.func the keys of the general way have no memory of their own
    for call in (lambda f: torch.func.jvp(f, (vals,), (tang,)), lambda f: torch.func.grad(f)(vals)):
        with pytest.raises(RuntimeError):
            call(lambda v: sort_unique_sum(keys, v, key_bits=8)[1].sum())
    v = vals.clone().requires_grad_()
    sort_unique_sum(keys, v, key_bits=8)[1].sum().backward()
    assert torch.all(v.grad == 1)


def test_values_that_torch_negates_on_reading(cuda_device):
    from ps_lite_b200.ops.keys import sort_unique_sum
    keys = torch.tensor([1, 0, 1], device=cuda_device)
    vals = torch._neg_view(torch.tensor([1.0, 2.0, 4.0], device=cuda_device))
    assert vals.is_neg() and sort_unique_sum(keys, vals, key_bits=8)[1].tolist() == [-2.0, -5.0]


def test_forms_that_stay_refused(cuda_device):
    """All refused by the host."""
    from ps_lite_b200.ops.keys import sort_unique_sum
    keys, vals = torch.arange(6, device=cuda_device), torch.ones(6, device=cuda_device)
    for k, v in ((keys.view(2, 3), vals), (keys.view(2, 3).t(), vals), (keys, vals.cpu()),
                 (keys.cpu(), vals), (keys.int(), vals)):
        with pytest.raises((AssertionError, RuntimeError, IndexError)):
            sort_unique_sum(k, v, key_bits=8)
