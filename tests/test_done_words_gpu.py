"""Requests of one rank whose kernel itself tells the host that it is done: what a request has written
is there for another stream once it has been waited for, from one CTA to more than count themselves,
with more requests in flight than there are words, and from several threads."""
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
    for key, n in enumerate([1, 1024, 1025, 37 * 1024, 16384 * 1024, 16384 * 1024 + 1]):
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
