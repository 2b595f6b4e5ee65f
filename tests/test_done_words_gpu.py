"""Requests of one rank whose kernel itself tells the host that it is done: what a request has written
is there for another stream, for a copy engine and for the host once it has been waited for, from one
CTA to more than count themselves, with more requests in flight than there are words, and from several
threads."""
import os
import subprocess
import sys
import textwrap

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(code, **env):
    head = f"import sys; sys.path.insert(0, {ROOT!r})\n"
    r = subprocess.run([sys.executable, "-c", head + textwrap.dedent(code)], capture_output=True, text=True,
                       timeout=240, env=dict(os.environ, **env))
    assert r.returncode == 0 and "RAN" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]


DENSE = """
    import torch
    from ps_lite_b200 import kvstore
    from ps_lite_b200.parallel import ServerOptimizer
    ctx = kvstore.init(heap_bytes=1 << 30)
    kv = kvstore.KVStore(ctx)
    dev = ctx.device
    other = torch.cuda.Stream(dev)
    # CTAs of 1024 values: one, two, a few, as many as count themselves and one more
    for key, n in enumerate([1, 1024, 1025, 37 * 1024, 128 * 1024, 128 * 1024 + 1, 1 << 24]):
        kv.declare(key, n, optimizer=ServerOptimizer("sum"))
        grad, out = torch.ones(n, device=dev), torch.zeros(n, device=dev)
        torch.cuda.synchronize()
        for i in range(1, 200 if n < 100_000 else 30):
            kv.wait(kv.push_pull(key, grad, out))
            with torch.cuda.stream(other):   # not ordered behind the request's stream
                assert bool((out == i).all()), (n, i)
    # more in flight than there are words, on one tensor and on another
    n = 1025
    grad, outs = torch.ones(n, device=dev), [torch.zeros(n, device=dev) for _ in range(200)]
    ts = [kv.push_pull(2, grad, o) for o in outs]
    for t in reversed(ts):
        kv.wait(t)
    with torch.cuda.stream(other):
        first = outs[0][0].item()
        assert all(bool((o == first + i).all()) for i, o in enumerate(outs))
    kvstore.finalize()
    print("RAN")
"""


def test_dense_requests(cuda_device):
    _run(DENSE)


def test_dense_requests_without_words(cuda_device):
    _run(DENSE, PSB200_SPIN_US="0")


def test_keyed_requests(cuda_device):
    _run("""
        import torch
        from ps_lite_b200 import kvstore
        ctx = kvstore.init(heap_bytes=1 << 30)
        dev = ctx.device
        other = torch.cuda.Stream(dev)
        for app, (width, var) in enumerate([(1, False), (8, False), (3, False), (5, True)], 7):
            ks = kvstore.KeyedStore(ctx, app, 1 << 20, 20000, width=width, kind="sum", var_len=var)
            for n in [1, 256, 1025, 9000, 20000]:
                keys = torch.arange(n, device=dev) * 7 + n % 5
                lens = torch.full((n,), width, device=dev, dtype=torch.int32) if var else None
                vals, out = torch.ones(n * width, device=dev), torch.zeros(n * width, device=dev)
                torch.cuda.synchronize()
                for i in range(1, 40):
                    if var:
                        ks.wait(ks.push(keys, vals, lens))
                        ks.wait(ks.pull(keys, out, torch.empty_like(lens)))
                    else:
                        ks.wait(ks.push_pull(keys, vals, out))
                    if i == 1:
                        torch.cuda.synchronize()
                        start = out.clone()
                    with torch.cuda.stream(other):
                        assert bool((out == start + (i - 1)).all()), (width, var, n, i)
        kvstore.finalize()
        print("RAN")
    """)


def test_requests_of_several_threads(cuda_device):
    _run("""
        import threading, torch
        from ps_lite_b200 import kvstore
        from ps_lite_b200.parallel import ServerOptimizer
        ctx = kvstore.init(heap_bytes=1 << 28)
        kv = kvstore.KVStore(ctx)
        dev, n, bad = ctx.device, 3000, []
        for key in range(6):
            kv.declare(key, n, optimizer=ServerOptimizer("sum"))
        def run(key):
            torch.cuda.set_device(dev)
            with torch.cuda.stream(torch.cuda.Stream(dev)):
                grad, out = torch.ones(n, device=dev), torch.zeros(n, device=dev)
                for i in range(1, 300):
                    kv.wait(kv.push_pull(key, grad, out))
                    if i % 37 == 0 and not bool((out == i).all()):
                        bad.append((key, i))
        threads = [threading.Thread(target=run, args=(k,)) for k in range(6)]
        for t in threads: t.start()
        for t in threads: t.join()
        assert not bad, bad
        kvstore.finalize()
        print("RAN")
    """)


def test_copies_that_follow_no_event(cuda_device):
    """Another stream's copy engine takes the output to the host: nothing orders it behind the request
    but the host, which has waited for that."""
    _run("""
        import torch
        from ps_lite_b200 import kvstore
        from ps_lite_b200.parallel import ServerOptimizer
        ctx = kvstore.init(heap_bytes=1 << 30)
        kv, dev = kvstore.KVStore(ctx), ctx.device
        other = torch.cuda.Stream(dev)
        def reads(n, request, wait, out, step):
            host = torch.zeros(n, pin_memory=True)
            torch.cuda.synchronize()
            first = None
            for i in range(300):
                wait(request())
                with torch.cuda.stream(other):
                    host.copy_(out, non_blocking=True)
                other.synchronize()
                first = host[0].item() if first is None else first
                assert bool((host == first + i * step).all()), (n, i)
        for key, n in enumerate([1, 1024, 1025, 37 * 1024, 128 * 1024, 128 * 1024 + 1]):
            kv.declare(key, n, optimizer=ServerOptimizer("sum"))
            grad, out = torch.ones(n, device=dev), torch.zeros(n, device=dev)
            reads(n, lambda: kv.push_pull(key, grad, out), kv.wait, out, 1)
        ks = kvstore.KeyedStore(ctx, 7, 1 << 20, 20000, width=8, kind="sum")
        for n in [1, 300, 20000]:
            keys = torch.arange(n, device=dev) * 7 + 1
            vals, out = torch.full((n * 8,), 2.0, device=dev), torch.zeros(n * 8, device=dev)
            ks.wait(ks.pull(keys, out))
            ks.wait(ks.push(keys, -out))           # (what a smaller n has left)
            reads(n * 8, lambda: ks.push_pull(keys, vals, out), ks.wait, out, 2)
        kvstore.finalize()
        print("RAN")
    """)


@pytest.mark.parametrize("kind", ["managed", "mapped", "managed pool", "mapped pool"])
def test_memory_that_the_host_reads(cuda_device, kind, tmp_path):
    """Tensors over memory that is the host's too: managed, mapped host memory, and pools of torch's
    allocator over either.  The host reads it as soon as it has waited.  What is host memory goes the
    way of host memory, whoever has made the tensor: 64 MiB both ways in slices."""
    source, lib = tmp_path / "managed.cc", tmp_path / "managed.so"
    source.write_text("""
        #include <cuda_runtime.h>
        extern "C" void* take(long size, int, cudaStream_t) {
          void* p = nullptr;
          return cudaMallocManaged(&p, size) == cudaSuccess ? p : nullptr;
        }
        extern "C" void give(void* p, long, int, cudaStream_t) { cudaFree(p); }
        extern "C" void* mapped(long size, int, cudaStream_t) {
          void* p = nullptr;
          return cudaHostAlloc(&p, size, cudaHostAllocMapped) == cudaSuccess ? p : nullptr;
        }
        extern "C" void unmapped(void* p, long, int, cudaStream_t) { cudaFreeHost(p); }
    """)
    subprocess.run(["nvcc", "-shared", "-Xcompiler", "-fPIC", "-x", "cu", str(source), "-o", str(lib)], check=True)
    _run(f"""
        import ctypes, os, numpy as np, torch
        from ps_lite_b200 import host, kvstore
        from ps_lite_b200.parallel import ServerOptimizer
        ctx = kvstore.init(heap_bytes=1 << 29)
        kv, dev, kind = kvstore.KVStore(ctx), ctx.device, {kind!r}
        lib, names = ctypes.CDLL({str(lib)!r}), ("take", "give") if "managed" in kind else ("mapped", "unmapped")
        make = getattr(lib, names[0])
        make.restype, make.argtypes = ctypes.c_void_p, [ctypes.c_long, ctypes.c_int, ctypes.c_void_p]
        if "pool" in kind:
            own = torch.cuda.memory.CUDAPluggableAllocator({str(lib)!r}, *names)
            pool = torch.cuda.MemPool(own.allocator())
        def tensor(n):
            if "pool" in kind:
                with torch.cuda.use_mem_pool(pool):
                    return torch.zeros(n, device=dev)
            class Array:
                __cuda_array_interface__ = dict(shape=(n,), typestr="<f4", data=(make(4 * n, 0, None), False),
                                                version=3)
            return torch.as_tensor(Array(), device=dev)
        def launches(key, grad, out):
            before = host.lib().psnvl_launches()
            kv.wait(kv.push_pull(key, grad, out))
            return host.lib().psnvl_launches() - before
        for key, n in enumerate([1000, 100_000, 1_000_000, 1 << 24]):
            kv.declare(key, n, optimizer=ServerOptimizer("sum"))
            grad, out = tensor(n).fill_(1.0), tensor(n).zero_()
            seen = np.ctypeslib.as_array(ctypes.cast(out.data_ptr(), ctypes.POINTER(ctypes.c_float)), (n,))
            torch.cuda.synchronize()
            for i in range(1, 60 if n < 1 << 24 else 4):
                kv.wait(kv.push_pull(key, grad, out))
                assert (seen == i).all(), (n, i)
        torch.cuda.synchronize()
        like = torch.ones(n, pin_memory=True) if "mapped" in kind else torch.ones(n, device=dev)
        torch.cuda.synchronize()
        assert launches(key, grad, out) == launches(key, like, torch.empty_like(like, pin_memory=like.is_pinned()))
        kvstore.finalize()
        print("RAN", flush=True)
        os._exit(0)   # (the tensors' memory has no owner)
    """)
