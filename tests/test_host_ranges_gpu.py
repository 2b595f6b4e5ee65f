"""psdev_rt_host_mapped: which ranges of host memory a kernel may access (asked, never accessed)."""
import ctypes as C
import mmap

import pytest
import torch

pytestmark = pytest.mark.gpu


def _mapped(p, n):
    from ps_lite_b200 import _lib
    fn = _lib.device_lib().psdev_rt_host_mapped
    fn.argtypes, fn.restype = [C.c_void_p, C.c_size_t, C.c_void_p], C.c_int
    dev = C.c_void_p()
    got = fn(p, n, C.byref(dev))
    assert not got or dev.value
    return bool(got)


def test_ranges_inside_and_across_registrations(cuda_device):
    torch.zeros(1, device=cuda_device)
    rt, page = torch.cuda.cudart(), mmap.PAGESIZE
    area = mmap.mmap(-1, 16 * page)
    base = C.addressof(C.c_char.from_buffer(area))
    # pages 0..3 and 8..11 are registered one by one, 4..7 are ordinary memory
    assert int(rt.cudaHostRegister(base, 4 * page, 0)) == 0
    assert int(rt.cudaHostRegister(base + 8 * page, 4 * page, 0)) == 0
    try:
        for first in (0, 8):
            at = base + first * page
            for off, n in ((0, 1), (0, 4 * page), (1, 4 * page - 1), (4 * page - 1, 1), (page + 7, 1000)):
                assert _mapped(at + off, n), (first, off, n)
            for off, n in ((0, 4 * page + 1), (1, 4 * page), (4 * page - 1, 2), (page, 0)):
                assert not _mapped(at + off, n), (first, off, n)
        assert not _mapped(base, 12 * page)          # both ends registered, a hole between them
        assert not _mapped(base + 3 * page, 6 * page)
        assert not _mapped(base + 5 * page, page)    # ordinary memory
        assert not _mapped(base + 5 * page, 4 * page)
    finally:
        rt.cudaHostUnregister(base)
        rt.cudaHostUnregister(base + 8 * page)


def test_tensors(cuda_device):
    t = torch.zeros(100_003).pin_memory()
    assert _mapped(t.data_ptr(), 4 * t.numel()) and _mapped(t[1:].data_ptr(), 4 * (t.numel() - 1))
    assert not _mapped(torch.zeros(100).data_ptr(), 400)
    assert not _mapped(torch.zeros(100, device=cuda_device).data_ptr(), 400)
