"""What the native forms of the Python calls refuse, before anything reaches a GPU: the functions that
they would call are addresses nobody must jump to."""
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
