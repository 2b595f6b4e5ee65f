"""sort_keys around the number of chunks up to which the scatter kernel adds up the digit counts itself
(32 chunks of 4096 keys): against torch.sort, stable, with and without the permutation."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [4097, 8192, 16_385, 31 * 4096, 32 * 4096 - 1, 32 * 4096, 32 * 4096 + 1, 33 * 4096 + 5])
@pytest.mark.parametrize("bits,spread", [(16, 5), (30, 1 << 30), (64, 1 << 62), (8, 1)])
def test_sorted_and_stable(cuda_device, n, bits, spread):
    from ps_lite_b200.ops.keys import sort_keys
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n + bits)
    keys = torch.randint(0, spread, (n,), device=cuda_device, generator=g)
    want, order = torch.sort(keys, stable=True)
    got, perm = sort_keys(keys.clone(), bits, return_perm=True)
    assert torch.equal(got, want) and torch.equal(perm.long(), order)
    assert torch.equal(sort_keys(keys.clone(), bits)[0], want)


@pytest.mark.parametrize("n,each", [(4097, 2), (1 << 16, 2), ((1 << 16) + 1, 2), (80 << 10, 2), (96 << 10, 2),
                                    (32 * 4096, 2), (32 * 4096 + 1, 3)])
def test_launches_per_pass(cuda_device, n, each):
    """No scan where the scatter adds up the counts."""
    from ps_lite_b200 import _lib
    from ps_lite_b200.ops.keys import sort_keys
    lib = _lib.device_lib()
    keys = torch.arange(n, device=cuda_device).flip(0).contiguous()
    before = lib.psdev_launch_count()
    assert torch.equal(sort_keys(keys, 24)[0], torch.arange(n, device=cuda_device))
    assert lib.psdev_launch_count() - before == 3 * each
