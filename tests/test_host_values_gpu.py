"""KVStore requests on pinned host tensors, one rank: sizes below and above the limits up to which
the kernel accesses host memory itself (48 MiB both ways, 16 MiB one way), arrays of any alignment,
requests with one side on the device, pageable memory, and tensors of the wrong shape."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("gdt,odt", [("float32", "float32"), ("bfloat16", "bfloat16"),
                                     ("bfloat16", "float32")])
def test_host_tensors(cuda_device, gdt, odt):
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import torch
        from ps_lite_b200 import kvstore, host
        from ps_lite_b200.parallel import ServerOptimizer
        gdt, odt = torch.%s, torch.%s
        ctx = kvstore.init(heap_bytes=1 << 30)
        kv = kvstore.KVStore(ctx)
        L = host.lib()
        for key, n in enumerate((1, 1023, 300_003, 4_400_001, 13_000_008)):
            t = kv.declare(key, n, grad_dtype=gdt, out_dtype=odt, optimizer=ServerOptimizer("sum"))
            # small whole numbers: sums are exact in every type
            grad = (torch.arange(n) %% 5 - 2).to(gdt)
            want = torch.zeros(n)
            for shift, pinned in ((0, True), (1, True), (3, True), (0, False)):
                src, dst = torch.zeros(n + shift, dtype=gdt), torch.full((n + shift,), 9., dtype=odt)
                if pinned:
                    src, dst = src.pin_memory(), dst.pin_memory()
                src[shift:] = grad
                a = L.psnvl_launches()
                kv.wait(kv.push_pull(key, src[shift:], dst[shift:]))
                launches = L.psnvl_launches() - a
                big = n * max(src.element_size(), dst.element_size()) > 48 << 20
                sliced = big if pinned else n * src.element_size() > 4 << 20
                assert (launches > 1) == sliced, (n, shift, pinned, launches)
                want += grad.float()
                assert torch.equal(dst[shift:].float(), want) and torch.all(dst[:shift] == 9.)
                assert torch.equal(t.weight[:n].float().cpu(), want)
                kv.wait(kv.push(key, src[shift:]))
                want += grad.float()
                kv.wait(kv.pull(key, dst[shift:]))
                assert torch.equal(dst[shift:].float(), want)
                # one side on the device
                dev = torch.empty(n, dtype=odt, device=ctx.device)
                kv.wait(kv.push_pull(key, src[shift:], dev))
                want += grad.float()
                assert torch.equal(dev.float().cpu(), want)
                kv.wait(kv.push_pull(key, grad.to(ctx.device), dst[shift:]))
                want += grad.float()
                assert torch.equal(dst[shift:].float(), want)
                if n > 4_000_000 and shift == 1:
                    break
            for wrong in (torch.zeros(n + 1, dtype=gdt), torch.zeros(n, dtype=torch.int32)):
                try:
                    kv.push(key, wrong)
                    raise SystemExit("accepted")
                except ValueError:
                    pass
            for call in (lambda: kv.push(key, torch.zeros(n, 2, dtype=gdt)[:, 0] if n > 1 else
                                         torch.zeros(2, dtype=gdt)),
                         lambda: kv.pull(key, torch.zeros(n + 8, dtype=odt))):
                try:
                    call()
                    raise SystemExit("accepted")
                except ValueError:
                    pass
        kvstore.finalize(); print("HOST_OK")
    """ % (ROOT, gdt, odt)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "HOST_OK" in r.stdout, (r.stdout + r.stderr)[-3000:]
