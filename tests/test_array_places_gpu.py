"""One rank: requests whose arrays are not all on the GPU of the table go through the table's buffers."""
import ctypes as C
import os
import subprocess
import sys

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_where_memory_is(cuda_device):
    from ps_lite_b200 import _lib
    fn = _lib.device_lib().psdev_rt_memory
    fn.argtypes, fn.restype = [C.c_void_p, C.POINTER(C.c_int)], C.c_int
    dev = C.c_int(-1)
    for d in range(torch.cuda.device_count()):
        assert fn(torch.zeros(100, device=f"cuda:{d}")[7:].data_ptr(), C.byref(dev)) == 1
        assert dev.value == d
    assert fn(torch.zeros(100).data_ptr(), C.byref(dev)) == 0
    assert fn(torch.zeros(100).pin_memory().data_ptr(), C.byref(dev)) == 0


CODE = """if 1:
    import sys; sys.path.insert(0, %r)
    import torch
    from ps_lite_b200 import host, kvstore
    from ps_lite_b200.parallel import ServerOptimizer
    places = %r
    ctx = kvstore.init(heap_bytes=256 << 20)
    L = host.lib()
    def put(t, where):
        return t.pin_memory() if where == "pinned" else t.to(where)
    # a keyed table: keys on the device, the other arrays wherever
    for var_len in (False, True):
        store = kvstore.KeyedStore(ctx, 1 + var_len, 1 << 16, 5000, width=4, kind="sum", var_len=var_len)
        n = 3001
        keys = (torch.randperm(1 << 16)[:n].sort().values).to(ctx.device)
        lens = torch.arange(n, dtype=torch.int32) %% 4 + 1 if var_len else None
        count = int(lens.sum()) if var_len else 4 * n
        vals = torch.randint(-50, 50, (count,)).float()
        want = torch.zeros(count)
        for a in places:
            for b in places:
                v, o = put(vals, a), put(torch.full((count,), 9.0), b)
                l = put(lens, b) if var_len else None
                torch.cuda.synchronize()
                ts = L.ps_capi_bworker_keyed_request(
                    store.worker, 1, 1, keys.data_ptr(), n, v.data_ptr(), 4 * count, o.data_ptr(),
                    4 * count, l.data_ptr() if var_len else None, None, 0)
                assert ts >= 0 and L.ps_capi_bworker_wait(store.worker, ts) >= 0, (a, b)
                torch.cuda.synchronize()
                want += vals
                assert torch.equal(o.cpu(), want), (var_len, a, b)
                o = put(torch.full((count,), 9.0), b)
                l = put(torch.zeros(n, dtype=torch.int32), a) if var_len else None
                torch.cuda.synchronize()
                ts = L.ps_capi_bworker_keyed_request(
                    store.worker, 0, 1, keys.data_ptr(), n, None, 0, o.data_ptr(), 4 * count, None,
                    l.data_ptr() if var_len else None, 0)
                assert ts >= 0 and L.ps_capi_bworker_wait(store.worker, ts) >= 0, (a, b)
                torch.cuda.synchronize()
                assert torch.equal(o.cpu(), want), (var_len, a, b)
                assert not var_len or torch.equal(l.cpu(), lens)
    # a dense tensor
    kv = kvstore.KVStore(ctx)
    n = 50_001
    t = kv.declare(0, n, optimizer=ServerOptimizer("sum"))
    grad, want = torch.randint(-50, 50, (n,)).float(), torch.zeros(n)
    for a in places:
        for b in places:
            g, o = put(grad, a), put(torch.zeros(n), b)
            torch.cuda.synchronize()
            kv.wait(kv.push_pull(0, g, o))
            want += grad
            torch.cuda.synchronize()
            assert torch.equal(o.cpu(), want), (a, b)
    kvstore.finalize(); print("PLACES_OK")
"""


def _run(places, code=CODE):
    r = subprocess.run([sys.executable, "-c", code % (ROOT, places)], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0 and "PLACES_OK" in r.stdout, (r.stdout + r.stderr)[-3000:]


def test_host_and_device(cuda_device):
    _run(["cuda:0", "cpu", "pinned"])


def test_a_command_says_nothing_about_arrays(cuda_device):
    """The number that once told the plane not to ask where the arrays of a request are."""
    code = CODE.replace("None, None, 0)", "None, None, 0x48455245)").replace("else None, 0)", "else None, 0x48455245)")
    code = code.replace("kv.wait(kv.push_pull(0, g, o))", "kv.wait(kv._request(0, True, True, g, o, cmd=0x48455245))")
    assert code.count("0x48455245") == 3
    _run(["cuda:0", "cpu", "pinned"], code)


def test_two_gpus(cuda_device):
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    _run(["cuda:0", "cuda:1"])
