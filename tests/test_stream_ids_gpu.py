"""Streams with one handle that are not one stream: the per-thread default stream of two threads.
Requests on one tensor from both are served one after the other."""
import ctypes as C
import os
import subprocess
import sys
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PER_THREAD = 2   # cudaStreamPerThread


def _id(handle):
    from ps_lite_b200 import _lib
    fn = _lib.device_lib().psdev_rt_stream_id
    fn.argtypes, fn.restype = [C.c_void_p, C.POINTER(C.c_uint64)], C.c_int
    out = C.c_uint64()
    assert fn(handle, C.byref(out)) == 0
    return out.value


def test_ids_tell_streams_apart(cuda_device):
    torch.zeros(1, device=cuda_device)
    a, b = torch.cuda.Stream(cuda_device), torch.cuda.Stream(cuda_device)
    assert _id(a.cuda_stream) == _id(a.cuda_stream) != _id(b.cuda_stream)
    ids = [_id(0), _id(PER_THREAD), _id(PER_THREAD)]
    t = threading.Thread(target=lambda: (torch.cuda.set_device(cuda_device), ids.append(_id(PER_THREAD))))
    t.start()
    t.join()
    assert ids[1] == ids[2] and len({ids[0], ids[1], ids[3]}) == 3 and all(ids)


def test_requests_of_two_threads_on_their_default_streams(cuda_device):
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import threading, torch
        from ps_lite_b200 import kvstore
        from ps_lite_b200.parallel import ServerOptimizer
        ctx = kvstore.init(heap_bytes=1 << 30)
        kv = kvstore.KVStore(ctx)
        n = 8 << 20
        t = kv.declare(0, n, optimizer=ServerOptimizer("sum"))
        ones = torch.ones(n, device=ctx.device)
        torch.cuda.synchronize()
        gate = threading.Barrier(2)
        lock = threading.Lock()   # requests are handed over one at a time, not waited for
        def run():
            torch.cuda.set_device(ctx.device)
            with torch.cuda.stream(torch.cuda.ExternalStream(%d, device=ctx.device)):
                for _ in range(40):
                    gate.wait()
                    with lock:
                        kv.push(0, ones)
        threads = [threading.Thread(target=run) for _ in range(2)]
        for x in threads: x.start()
        for x in threads: x.join()
        kv.wait_all()
        kv.wait(kv.pull(0))
        assert torch.all(t.weight[:n] == 80.0), t.weight[:n].unique()
        kvstore.finalize(); print("STREAMS_OK")
    """ % (ROOT, PER_THREAD)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "STREAMS_OK" in r.stdout, (r.stdout + r.stderr)[-3000:]
