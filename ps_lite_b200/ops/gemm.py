"""bf16 GEMM on the tcgen05 tensor cores, alone or fused with the pull of its weights."""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _lib


class _Native:
    """The native calls and the addresses they are given, resolved at the first use."""

    def __getattr__(self, name):
        lib, ext = _lib.device_lib(), _lib.torch_ext()
        self.gemm_fn = C.cast(lib.psdev_gemm_bf16, C.c_void_p).value
        self.pull_fn = C.cast(lib.psdev_pull_gemm_bf16, C.c_void_p).value
        self.linear, self.pull_linear = ext.linear, ext.pull_linear
        return self.__dict__[name]


_native = _Native()


def gemm_status(device) -> int:
    """Error word of the last GEMM launches on ``device`` (0 = none); synchronises."""
    st = C.c_int32()
    with torch.cuda.device(device):
        _lib.check(_lib.device_lib().psdev_gemm_status(C.byref(st)), "psdev_gemm_status")
    return st.value


def linear_bf16(x: torch.Tensor, w: torch.Tensor, out: Optional[torch.Tensor] = None,
                num_ctas: int = 0, timeout_s: float = 2.0) -> torch.Tensor:
    """``out[M,N] = x[M,K] @ w[N,K]^T`` (bf16 in, fp32 accumulate, bf16 out)."""
    got = _native.linear(_native.gemm_fn, x, w, out, num_ctas, int(timeout_s * 1e9))
    if type(got) is int:
        _lib.check(got, "psdev_gemm_bf16")
    return got


def pull_linear_bf16(table, w_offset: int, n_out: int, x: torch.Tensor,
                     out: Optional[torch.Tensor] = None, num_copy_ctas: int = 0,
                     num_ctas: int = 0, timeout_s: float = 2.0) -> torch.Tensor:
    """Pull ``W = table.weight[w_offset : w_offset + n_out*K]`` (viewed ``[n_out, K]``) from its
    owners and compute ``x @ W^T`` in the same kernel.

    Must follow, on the same stream, a ``table.push(..., publish=True)`` covering that range.
    Afterwards ``table.weight`` holds the complete W locally (for the backward pass).
    """
    assert table.out_dtype == torch.bfloat16
    got = _native.pull_linear(_native.pull_fn, table._world_at, table._table_at, int(w_offset),
                              n_out, x, out, num_copy_ctas, num_ctas, int(timeout_s * 1e9))
    if type(got) is int:
        _lib.check(got, "psdev_pull_gemm_bf16")
    return got


def fusion_pays(weight_bytes: int, world: int) -> bool:
    """Whether pulling a weight inside the GEMM that consumes it beats push+pull followed by
    the GEMM.  Measured (benchmarks/pull_gemm_bench.py): with a 128 MiB weight the fused form
    is 1.12-1.16x faster; with the 6 MiB QKV weight of BERT-large it is slower (0.96x on 2 GPUs,
    0.91x on 4: the cooperative launch and the per-panel waits cost more than the pull they
    hide).  The switch-over lies between; ``PSB200_FUSE_MIN_MB`` (default 32) sets it."""
    import os
    if world < 2:
        return False
    return weight_bytes >= int(os.environ.get("PSB200_FUSE_MIN_MB", "32")) << 20


class _PullLinearFn(torch.autograd.Function):
    """``x @ W^T`` where W is pulled from its owners inside the GEMM kernel.

    ``weight`` is the parameter whose storage is the table's weight slice: the kernel fills
    it while multiplying, so the backward pass can use it as an ordinary local tensor."""

    @staticmethod
    def forward(ctx, x, weight, table, w_offset):
        n_out, k = weight.shape
        x2 = x.reshape(-1, k).contiguous()
        out = pull_linear_bf16(table, w_offset, n_out, x2)
        ctx.save_for_backward(x2, weight)
        ctx.x_shape = x.shape
        return out.view(*x.shape[:-1], n_out)

    @staticmethod
    def backward(ctx, dy):
        x2, weight = ctx.saved_tensors
        dy2 = dy.reshape(-1, weight.shape[0])
        dx = (dy2 @ weight).view(ctx.x_shape)
        dw = dy2.t() @ x2
        return dx, dw, None, None


def pull_linear(x: torch.Tensor, weight: torch.nn.Parameter, table, w_offset: int) -> torch.Tensor:
    """Differentiable form of :func:`pull_linear_bf16` for a parameter stored in ``table``."""
    return _PullLinearFn.apply(x, weight, table, w_offset)
