"""psdev_copy_cast, with which gradient hooks copy: every value as torch casts it, and the bits of a
copy of one type, for arrays that begin anywhere."""
import pytest
import torch

TYPES = {"fp32": (torch.float32, 0, torch.int32), "bf16": (torch.bfloat16, 1, torch.int16)}


@pytest.mark.gpu
@pytest.mark.parametrize("source", TYPES)
@pytest.mark.parametrize("target", TYPES)
@pytest.mark.parametrize("n", [1, 7, 8, 9, 2047, 2048, 2049, 1_000_003])
def test_values(cuda_device, source, target, n):
    from ps_lite_b200 import _lib
    (st, si, bits), (tt, ti, _) = TYPES[source], TYPES[target]
    for begin_in, begin_out in [(0, 0), (1, 0), (8, 3), (8, 8)]:
        x = torch.randn(n + begin_in, device=cuda_device).to(st)[begin_in:]
        x[:: 97] = float("inf")
        x[1:: 101] = float("-inf")
        x[2:: 103] = 1e-41
        if st == tt:
            x.view(bits)[3:: 107] = 0x7FC1 if bits == torch.int16 else 0x7FC00123   # a NaN's payload
        out = torch.full((n + begin_out + 8,), 7.0, device=cuda_device, dtype=tt)
        rc = _lib.device_lib().psdev_copy_cast(
            x.data_ptr(), si, out.data_ptr() + begin_out * out.element_size(), ti, n,
            torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        got, want = out[begin_out:begin_out + n], x.to(tt)
        assert torch.equal(got.view(TYPES[target][2]), want.view(TYPES[target][2]))
        assert bool((out[:begin_out] == 7).all()) and bool((out[begin_out + n:] == 7).all())


@pytest.mark.parametrize("args", [(0, 2, 4), (2, 0, 4), (-1, 0, 4), (0, 0, -1)])
def test_what_is_refused(args):
    from ps_lite_b200 import _lib
    source, target, n = args
    assert _lib.device_lib().psdev_copy_cast(None, source, None, target, n, None) == -1
