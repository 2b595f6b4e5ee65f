"""Key-list utilities on the device: radix sort, unique, ordered match (merge-join).

Device counterparts of the reference's ``ParallelSort`` and ``ParallelOrderedMatch`` helpers
(include/ps/internal/parallel_sort.h:23-55, parallel_kv_match.h:29-120) and its ``AssignOp``
operators (assign_op.h:12-21)."""
from __future__ import annotations

import ctypes as C
from typing import Optional, Tuple

import torch

from .. import _lib

ASSIGN, PLUS, MINUS, TIMES, DIVIDE, AND, OR, XOR = range(8)


def sort_keys(keys: torch.Tensor, key_bits: int = 64, return_perm: bool = False,
              check: bool = False) -> Tuple[torch.Tensor, Optional[torch.Tensor]]:
    """Sort uint64 keys (stored as int64 bit patterns) ascending, in place; keys must be below
    ``2**key_bits``.  With ``return_perm`` also returns the stable permutation (int32 indices
    into the input).  ``check`` waits for the sort and raises if it failed."""
    assert keys.is_cuda and keys.dtype == torch.int64 and keys.is_contiguous()
    lib = _lib.device_lib()
    n = keys.numel()
    perm = torch.empty(n, dtype=torch.int32, device=keys.device) if return_perm else None
    nbytes = lib.psdev_sort_scratch_bytes(n, 1 if return_perm else 0)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device=keys.device)
    rc = lib.psdev_sort_keys(keys.data_ptr(), perm.data_ptr() if perm is not None else None, n,
                             key_bits, scratch.data_ptr(), nbytes,
                             torch.cuda.current_stream(keys.device).cuda_stream)
    _lib.check(rc, "psdev_sort_keys")
    if check:
        _lib.check(lib.psdev_sort_status(scratch.data_ptr(),
                                         torch.cuda.current_stream(keys.device).cuda_stream),
                   "psdev_sort_status")
    return keys, perm


class _Native:
    """The native call and the addresses it is given, resolved at the first use."""

    def __getattr__(self, name):
        lib, ext = _lib.device_lib(), _lib.torch_ext()
        self.fns = tuple(C.cast(f, C.c_void_p).value for f in (
            lib.psdev_unique_sum_scratch_bytes, lib.psdev_unique_sum_sort,
            lib.psdev_unique_sum_write))
        self.unique_sum = ext.unique_sum
        return self.__dict__[name]


_native = _Native()


def sort_unique_sum(keys: torch.Tensor, vals: torch.Tensor, key_bits: int = 64
                    ) -> Tuple[torch.Tensor, torch.Tensor]:
    """Turn arbitrary (key, value) pairs into the sorted unique keys a push needs, summing the
    values of repeated keys; keys must be below ``2**key_bits``.  fp32 values travel with the
    keys through the sort and are summed by a kernel of their own; other types take the sort
    permutation and torch's ``index_add_``.

    The values of a key are added up in a fixed tree, so that equal inputs have equal sums, bit for
    bit.  From 786 433 to 4 718 592 pairs (16 to 42 bits) the places in that tree also depend on the
    order in which the GPU serves lanes that count on one address: it has been the same from run to
    run, but nothing guarantees it."""
    if keys.is_cuda:
        got = _native.unique_sum(*_native.fns, keys, vals, key_bits)
        if type(got) is tuple:
            return got
        if got is not None:  # (None: another type, or a key wider than key_bits)
            _lib.check(got, "psdev_unique_sum")
    k = keys.clone()
    k, perm = sort_keys(k, key_bits, return_perm=True)
    v = vals[perm.long()]
    uk, inv = torch.unique_consecutive(k, return_inverse=True)
    out = torch.zeros(uk.numel(), dtype=vals.dtype, device=vals.device)
    out.index_add_(0, inv, v)
    return uk, out


def ordered_match(src_keys: torch.Tensor, src_vals: torch.Tensor, dst_keys: torch.Tensor,
                  dst_vals: torch.Tensor, op: int = ASSIGN, k: int = 1) -> int:
    """``dst_vals[j] op= src_vals[i]`` for every key in both sorted unique lists (``k`` values
    per key); returns how many keys matched."""
    assert src_vals.dtype == dst_vals.dtype and src_vals.dtype in (torch.float32, torch.int32)
    matched = torch.zeros(1, dtype=torch.int64, device=dst_vals.device)
    rc = _lib.device_lib().psdev_ordered_match(
        src_keys.data_ptr(), src_vals.data_ptr(), src_keys.numel(), dst_keys.data_ptr(),
        dst_vals.data_ptr(), dst_keys.numel(), k, op,
        0 if src_vals.dtype == torch.float32 else 1, matched.data_ptr(),
        torch.cuda.current_stream(dst_vals.device).cuda_stream)
    _lib.check(rc, "psdev_ordered_match")
    return int(matched.item())
