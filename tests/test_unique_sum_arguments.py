"""The second half of a sort of (key, value) pairs refuses what the first half refuses, before anything
reaches a GPU (the addresses here are never read)."""
import ctypes as C

import pytest


@pytest.fixture(scope="module")
def lib():
    from ps_lite_b200 import _lib
    return _lib.device_lib()


def _write(lib, n, key_bits):
    fn = lib.psdev_unique_sum_write
    return fn(C.c_void_p(1 << 20), C.c_int64(n), C.c_int(key_bits), C.c_int64(1),
              C.c_void_p(2 << 20), C.c_void_p(3 << 20), None)


@pytest.mark.parametrize("n", [1, 4096, 4097, 1 << 25])
@pytest.mark.parametrize("key_bits", [0, -1, -100, 65, 1 << 20])
def test_key_bits(lib, n, key_bits):
    assert _write(lib, n, key_bits) == -1  # PSDEV_ERR_ARG


@pytest.mark.parametrize("n,code", [(0, -1), (-1, -1), (1 << 30, -4), (1 << 40, -4)])
def test_items(lib, n, code):
    assert _write(lib, n, 30) == code
