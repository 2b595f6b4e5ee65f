"""Single-rank update kernel: arrays outside the arena, of any alignment and length, and pieces
with gradient arrays of their own give what the same values in the tensor's own buffers give --
the arithmetic per value is the same, so the results are compared bit for bit, and once against
the fp32 statement of the update."""
import ctypes as C

import pytest
import torch

from ps_lite_b200.utils.oracle import dense_update

pytestmark = pytest.mark.gpu


def _table(dev, n, gdt, odt, kind):
    from ps_lite_b200.parallel import DenseTable, ServerOptimizer, SymmetricHeap
    heap = SymmetricHeap(16 * n + (1 << 20), 0, 1, device=dev)
    t = DenseTable(heap, n, gdt, odt, optimizer=ServerOptimizer(kind, lr=0.05, eps=1e-6))
    g = torch.Generator(device=dev)
    g.manual_seed(n)
    w0 = torch.randn(n, device=dev, generator=g)
    t.load_master(w0)
    return heap, t, w0, g


def _direct(t, op, src, dst, n):
    from ps_lite_b200 import _lib
    t.step += 1
    lib = _lib.device_lib()
    _lib.check(lib.psdev_dense_op_direct(
        C.byref(t._world), C.byref(t._table), op, 0, t.n, C.byref(t._opt_struct()), 0, 0,
        torch.cuda.current_stream().cuda_stream, None if src is None else src.data_ptr(),
        None if dst is None else dst.data_ptr(), n), "direct")


@pytest.mark.parametrize("n", [1, 7, 8, 1023, 1024, 1025, 2048 + 9, 300_003])
@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("gdt,odt,kind", [(torch.float32, torch.float32, "sgd"),
                                          (torch.bfloat16, torch.bfloat16, "momentum"),
                                          (torch.bfloat16, torch.float32, "adam"),
                                          (torch.float32, torch.bfloat16, "adam")])
def test_arrays_outside_the_arena(cuda_device, n, shift, gdt, odt, kind):
    from ps_lite_b200 import _lib
    h1, a, w0, g = _table(cuda_device, n, gdt, odt, kind)
    h2, b, _, _ = _table(cuda_device, n, gdt, odt, kind)
    grad = torch.randn(n + shift, device=cuda_device, generator=g).to(gdt)[shift:]
    out = torch.full((n + shift + 8,), 7.0, device=cuda_device, dtype=odt)
    a.grad[:n].copy_(grad)
    a.push_pull()
    _direct(b, _lib.OP_PUSHPULL, grad, out[shift:], n)
    assert torch.equal(a.master, b.master) and torch.equal(a.weight, b.weight)
    assert torch.equal(out[shift:shift + n], a.weight[:n])
    assert torch.all(out[:shift] == 7.0) and torch.all(out[shift + n:] == 7.0)
    ref = dense_update(w0.clone(), [grad], kind, lr=0.05, momentum=0.9, eps=1e-6, step=1,
                       s1=torch.zeros(n, device=cuda_device), s2=torch.zeros(n, device=cuda_device))
    torch.testing.assert_close(b.master[:n], ref, rtol=2e-5, atol=2e-5)
    # push alone, then pull alone
    a.push()
    a.pull()
    _direct(b, _lib.OP_PUSH, grad, None, n)
    out.fill_(7.0)
    b.step -= 1
    _direct(b, _lib.OP_PULL, None, out[shift:], n)
    assert torch.equal(a.master, b.master) and torch.equal(out[shift:shift + n], a.weight[:n])
    h1.close()
    h2.close()


@pytest.mark.parametrize("gdt,sdt", [(torch.bfloat16, torch.float32), (torch.float32, torch.float32),
                                     (torch.bfloat16, torch.bfloat16),
                                     (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("pieces", [1, 2, 63, 64, 65, 200])
def test_pieces_with_their_own_gradients(cuda_device, gdt, sdt, pieces):
    """More pieces than one launch carries, pieces inside one tile and over several, a length
    that is no multiple of 8, and one piece whose gradient is in the arena."""
    from ps_lite_b200 import _lib
    lens = [1 + (i * 977) % 3001 for i in range(pieces)]
    begins, n = [], 0
    for k in lens:
        begins.append(n)
        n += (k + 7) & ~7
    h1, a, _, g = _table(cuda_device, n, gdt, torch.float32, "adam")
    h2, b, _, _ = _table(cuda_device, n, gdt, torch.float32, "adam")
    segs = (_lib.Seg * pieces)()
    grads = []
    for i, (s, at, k) in enumerate(zip(segs, begins, lens)):
        shift = i % 3
        x = torch.randn(k + shift, device=cuda_device, generator=g).to(sdt)[shift:]
        grads.append(x)
        a.grad[at:at + k].copy_(x)
        s.begin, s.end, s.n_valid = at, at + ((k + 7) & ~7), at + k
        s.priority, s.src, s.dtype = i % 5, x.data_ptr(), 0 if sdt == torch.float32 else 1
    b.grad[begins[-1]:begins[-1] + lens[-1]].copy_(grads[-1])
    segs[pieces - 1].src = None
    a.push_pull()
    b.step += 1
    _lib.check(_lib.device_lib().psdev_dense_op_segs(
        C.byref(b._world), C.byref(b._table), _lib.OP_PUSHPULL, segs, pieces,
        C.byref(b._opt_struct()), 0, 0, torch.cuda.current_stream().cuda_stream), "segs")
    assert torch.equal(a.master, b.master) and torch.equal(a.weight, b.weight)
    h1.close()
    h2.close()


def test_request_whose_arrays_overlap(cuda_device):
    """KVStore: output on top of the gradients, of another type and shifted, and the tensor's own
    buffers handed in as arrays: as if the values had been copied first."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    code = """if 1:
        import sys; sys.path.insert(0, %r)
        import torch
        from ps_lite_b200 import kvstore
        from ps_lite_b200.parallel import ServerOptimizer
        ctx = kvstore.init(heap_bytes=256 << 20)
        kv = kvstore.KVStore(ctx)
        n = 100_003
        t = kv.declare(0, n, grad_dtype=torch.bfloat16, optimizer=ServerOptimizer("sum"))
        raw = torch.zeros(2 * n + 8, device=ctx.device)
        for shift in (0, 3):
            t.master.zero_()
            grad = raw.view(torch.bfloat16)[2 * shift:2 * shift + n]
            grad.copy_(torch.arange(n, device=ctx.device) %% 128)
            want = grad.float()
            kv.wait(kv.push_pull(0, grad, raw[:n]))
            assert torch.equal(raw[:n], want), shift
        t2 = kv.declare(1, n, optimizer=ServerOptimizer("sum"))
        t2.grad[:n].fill_(2.0)
        kv.wait(kv.push_pull(1, t2.grad[:n], t2.grad[:n]))     # in place
        assert torch.all(t2.grad[:n] == 2.0) and torch.all(t2.weight[:n] == 2.0)
        kv.wait(kv.push_pull(1, t2.weight[:n], t2.weight[:n]))
        assert torch.all(t2.weight[:n] == 4.0)
        kvstore.finalize(); print("OVERLAP_OK")
    """ % root
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "OVERLAP_OK" in r.stdout, (r.stdout + r.stderr)[-3000:]
