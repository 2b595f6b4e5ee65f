"""What the native forms of the Python calls refuse, before anything reaches a GPU: the functions that
they would call are addresses nobody must jump to."""
import ctypes as C

import pytest
import torch


@pytest.fixture(scope="module")
def ext():
    from ps_lite_b200 import _lib
    return _lib.torch_ext()


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16)


def test_products_of_host_tensors_are_refused(ext):
    x, w = _bf16(64, 32), _bf16(16, 32)
    for args in ((x, w, None), (x, w, _bf16(64, 16)), (x.float(), w, None), (x, _bf16(16, 24), None)):
        with pytest.raises(AssertionError):
            ext.linear(0, *args, 0, 1)
    for args in ((x, None), (x, _bf16(64, 16)), (x.t(), None), (x.float(), None)):
        with pytest.raises(AssertionError):
            ext.pull_linear(0, 0, 0, 0, 16, *args, 0, 0, 1)


@pytest.mark.parametrize("limit", [0, 20 * 10 ** 9, -10 ** 9, (1 << 64) + 5])
def test_time_limits_wrap(ext, limit):
    """As ctypes hands them over: a negative limit of a caller stands for a wait without end."""
    got = []
    kind = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_void_p, C.c_int, C.c_int64, C.c_int64, C.c_void_p,
                       C.c_int, C.c_int, C.c_uint64, C.c_int, C.c_void_p)
    fn = kind(lambda *a: got.append(a) or 0)
    assert ext.dense_op(C.cast(fn, C.c_void_p).value, 8, 16, 3, 0, 64, 24, 1, 2, limit, 1, 40) == 0
    assert got == [(8, 16, 3, 0, 64, 24, 1, 2, C.c_uint64(limit).value, 1, 40)]
