"""GEMM for small products (one tile per cluster, K split over the CTAs) against fp32 matmul: ragged
tiles in M, N and K, fewer k-blocks than CTAs, more k-blocks than pipeline stages."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 64, 64), (127, 72, 72), (129, 136, 456),
                                   (64, 256, 256), (300, 1000, 1032), (256, 128, 4096),
                                   (2050, 520, 200)])
def test_matches_fp32_matmul(cuda_device, M, N, K, bn, split):
    from ps_lite_b200 import _lib
    from ps_lite_b200.ops.gemm import gemm_status, linear_bf16
    lib = _lib.device_lib()
    assert lib.psdev_gemm_config(1000 * split + bn) == 0
    try:
        torch.manual_seed(M + N + K)
        x = torch.randn(M, K, device=cuda_device).to(torch.bfloat16)
        w = (torch.randn(N, K, device=cuda_device) / K ** 0.5).to(torch.bfloat16)
        guard = torch.full((M + 2, N), 7.0, device=cuda_device, dtype=torch.bfloat16)
        out = linear_bf16(x, w, guard[1:M + 1])
        torch.cuda.synchronize()
        assert gemm_status(cuda_device) == 0
    finally:
        lib.psdev_gemm_config(0)
    ref = x.float() @ w.float().t()
    # fp32 sums of K products, then one rounding to bf16: 8 significant bits, so half a unit is at
    # most 2^-8 of the value
    bound = ref.abs() * 2.0 ** -8 * 1.01 + K * 2.0 ** -23 * (x.float().abs() @ w.float().abs().t())
    assert torch.all((out.float() - ref).abs() <= bound + 1e-6)
    assert torch.all(guard[0] == 7.0) and torch.all(guard[-1] == 7.0)


@pytest.mark.parametrize("bn", [64, 128])
@pytest.mark.parametrize("split", [1, 2, 4, 8])
@pytest.mark.parametrize("per", [2, 3, 4, 5])
@pytest.mark.parametrize("short", [0, 56])
def test_as_many_k_blocks_as_stages(cuda_device, per, short, bn, split):
    """Two to five k-blocks for each CTA of a cluster, where the form with two of them per stage begins;
    the last part one short."""
    test_matches_fp32_matmul(cuda_device, 200, 2 * bn + 8, 64 * per * split - short, bn, split)


def test_unknown_variants_are_refused(cuda_device):
    from ps_lite_b200 import _lib
    lib = _lib.device_lib()
    for bad in (64, 3064, 16064, 1032, -1):
        assert lib.psdev_gemm_config(bad) != 0
