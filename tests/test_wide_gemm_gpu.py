"""GEMM of large products (pairs of CTAs, 256 x 512 and 256 x 256 tiles) against fp32 matmul: ragged
tiles in M, N and K, one half of a wide tile outside N, fewer k-blocks than pipeline stages and than
the skew between the halves, several rounds, last rounds cut into two and four pieces along N."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [256, 512])
@pytest.mark.parametrize("M,N,K", [(256, 512, 64), (256, 256, 128), (257, 264, 72), (300, 520, 200),
                                   (1, 8, 8), (520, 1032, 456), (2000, 776, 1032),
                                   (2560, 2304, 128), (9728, 1024, 256), (9728, 1160, 320),
                                   (19456, 1000, 192)])
def test_matches_fp32_matmul(cuda_device, M, N, K, columns):
    from ps_lite_b200 import _lib
    from ps_lite_b200.ops.gemm import gemm_status, linear_bf16
    lib = _lib.device_lib()
    assert lib.psdev_gemm_config(2000 + columns) == 0
    try:
        torch.manual_seed(M + N + K)
        x = torch.randn(M, K, device=cuda_device).to(torch.bfloat16)
        w = (torch.randn(N, K, device=cuda_device) / K ** 0.5).to(torch.bfloat16)
        guard = torch.full((M + 2, N), 7.0, device=cuda_device, dtype=torch.bfloat16)
        outs = [linear_bf16(x, w, guard[1:M + 1]).clone() for _ in range(2)]
        torch.cuda.synchronize()
        assert gemm_status(cuda_device) == 0
    finally:
        lib.psdev_gemm_config(0)
    assert torch.equal(outs[0], outs[1])
    ref = x.float() @ w.float().t()
    # fp32 sums of K products, then one rounding to bf16: 8 significant bits, so half a unit is at
    # most 2^-8 of the value
    bound = ref.abs() * 2.0 ** -8 * 1.01 + K * 2.0 ** -23 * (x.float().abs() @ w.float().abs().t())
    assert torch.all((outs[0].float() - ref).abs() <= bound + 1e-6)
    assert torch.all(guard[0] == 7.0) and torch.all(guard[-1] == 7.0)


def test_follows_the_kernel_before_it(cuda_device):
    """The kernel may start before its predecessor ends: it must read what that one wrote."""
    from ps_lite_b200.ops.gemm import linear_bf16
    torch.manual_seed(1)
    for m, n in ((2048, 1024), (256, 256)):
        x = torch.randn(m, n, device=cuda_device).to(torch.bfloat16)
        eye = torch.eye(n, device=cuda_device).to(torch.bfloat16)
        y = x
        for _ in range(20):  # products with the identity: exact, each reads the one before
            y = linear_bf16(y, eye) + 1.0 - 1.0 if _ == 7 else linear_bf16(y, eye)
        z = x.clone()
        z = z + 1.0 - 1.0
        assert torch.equal(y, z)
