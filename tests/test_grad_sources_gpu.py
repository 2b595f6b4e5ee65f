"""Where the native hooks of DistributedOptimizer on one rank find a gradient: memory that belongs to
the gradient alone is read in place, memory that somebody else can write is copied by the hook."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class _FromWorkspace(torch.autograd.Function):
    """A layer whose backward makes its weight gradient in a workspace that all layers share."""

    @staticmethod
    def forward(ctx, x, p, value, ws):
        ctx.value, ctx.ws, ctx.shape = value, ws, p.shape
        return x.view_as(x)

    @staticmethod
    def backward(ctx, g):
        part = ctx.ws[:ctx.shape.numel()]
        part.fill_(ctx.value)
        return g, part.view(ctx.shape), None, None


def _optimizer(dev, params, gdt, overlap=True, batch_bytes=1 << 22, kind="sgd"):
    from ps_lite_b200.parallel import ServerOptimizer, SymmetricHeap
    from ps_lite_b200.parallel.optimizer import DistributedOptimizer
    n = sum((p.numel() + 7) & ~7 for p in params)
    heap = SymmetricHeap(8 * n + (1 << 20), 0, 1, device=dev)
    return heap, DistributedOptimizer(params, heap, ServerOptimizer(kind, lr=0.5, momentum=0.5),
                                      grad_dtype=gdt, overlap=overlap, batch_bytes=batch_bytes)


# whole numbers below 256 times powers of two: exact in bf16 and fp32
@pytest.mark.parametrize("batch_bytes", [1, 1 << 22])
@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("wdt,gdt", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16),
                                     (torch.float32, torch.float32), (torch.bfloat16, torch.float32)])
def test_workspace_written_again_for_the_next_layer(cuda_device, wdt, gdt, overlap, batch_bytes):
    shapes = [(1,), (9, 5), (1 << 18,), (513, 1025), (7,)]
    params = [torch.nn.Parameter(torch.zeros(s, device=cuda_device, dtype=wdt)) for s in shapes]
    heap, dopt = _optimizer(cuda_device, params, gdt, overlap, batch_bytes)
    ws = torch.zeros(513 * 1025, device=cuda_device, dtype=wdt)
    for step in range(3):
        x = torch.ones(1, device=cuda_device, requires_grad=True)
        for i, p in enumerate(params):
            x = _FromWorkspace.apply(x, p, 2.0 * (i + 1), ws)
        x.sum().backward()
        ws.fill_(99.0)      # ... and once more before the step ends
        dopt.step()
        for i, p in enumerate(params):
            assert torch.all(p == -(step + 1.0) * (i + 1)), (step, i)
    assert dopt._native.staged == 3 * len(params)
    dopt.close()
    heap.close()


def test_gradients_of_ordinary_layers_are_read_in_place(cuda_device):
    torch.manual_seed(1)
    net = torch.nn.Sequential(torch.nn.Conv2d(3, 8, 3), torch.nn.BatchNorm2d(8), torch.nn.Flatten(),
                              torch.nn.Linear(8 * 36, 40), torch.nn.LayerNorm(40),
                              torch.nn.Linear(40, 5, bias=False)).to(cuda_device)
    heap, dopt = _optimizer(cuda_device, list(net.parameters()), torch.float32)
    net(torch.randn(4, 3, 8, 8, device=cuda_device)).pow(2).sum().backward()
    dopt.step()
    assert dopt._native.staged == 0
    dopt.close()
    heap.close()


def test_gradients_that_somebody_keeps_are_copied(cuda_device):
    """... by a hook of the program, in a tensor that it hands over itself, or as a view."""
    shape = (40, 50)
    kept = []
    params = [torch.nn.Parameter(torch.zeros(shape, device=cuda_device)) for _ in range(4)]
    heap, dopt = _optimizer(cuda_device, params, torch.float32)
    params[0].register_post_accumulate_grad_hook(lambda p: kept.append(p.grad))
    params[1].grad = torch.zeros(shape, device=cuda_device)
    kept.append(params[1].grad)
    params[2].register_hook(lambda g: kept.append(g.view(-1)))
    two = torch.full(shape, 2.0, device=cuda_device)
    sum((p * two).sum() for p in params).backward()
    for t in kept:
        t.fill_(77.0)
    dopt.step()
    for p in params:
        assert torch.all(p == -1.0)
    assert 2 <= dopt._native.staged <= 3   # (autograd itself may copy what a tensor hook keeps)
    dopt.close()
    heap.close()


@pytest.mark.parametrize("kind", ["sgd", "momentum"])
@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("batch_bytes", [1, 4096, 1 << 22])
@pytest.mark.parametrize("gdt", [torch.float32, torch.bfloat16])
def test_two_backward_passes_before_a_step(cuda_device, gdt, batch_bytes, overlap, kind):
    """Every gradient is an update of its own, in the order of the passes: small and large tensors,
    one of them with gradients that go through the table's buffer (channels_last)."""
    shapes = [(3,), (1025,), (16, 8, 5, 3), (700_001,)]
    params = [torch.nn.Parameter(torch.zeros(s, device=cuda_device)) for s in shapes]
    want, speed = [0.0] * len(shapes), [0.0] * len(shapes)
    heap, dopt = _optimizer(cuda_device, params, gdt, overlap, batch_bytes, kind)
    for step in range(2):
        for value in (2.0, 6.0, 2.0):
            coef = [torch.full(s, value * (i + 1), device=cuda_device) for i, s in enumerate(shapes)]
            coef[2] = coef[2].contiguous(memory_format=torch.channels_last)
            sum((p * c).sum() for p, c in zip(params, coef)).backward()
            for i in range(len(shapes)):
                speed[i] = value * (i + 1) + (0.5 * speed[i] if kind == "momentum" else 0.0)
                want[i] -= 0.5 * speed[i]
        dopt.step()
        for p, w in zip(params, want):
            assert torch.all(p == w), (step, p.shape)   # halves and whole numbers: exact in fp32
    dopt.close()
    heap.close()


def test_pieces_that_overlap_are_refused(cuda_device):
    import ctypes as C

    from ps_lite_b200 import _lib
    from ps_lite_b200.parallel import DenseTable, ServerOptimizer, SymmetricHeap
    heap = SymmetricHeap(1 << 20, 0, 1, device=cuda_device)
    t = DenseTable(heap, 4096, optimizer=ServerOptimizer("sum"))
    for ranges, ok in (([(0, 64), (64, 128), (256, 512)], True), ([(64, 128), (0, 72)], False),
                       ([(512, 1024), (0, 64), (48, 56)], False), ([(8, 16), (8, 16)], False),
                       ([(256, 512), (64, 64), (0, 256)], True)):
        segs = (_lib.Seg * len(ranges))()
        for s, (b, e) in zip(segs, ranges):
            s.begin, s.end, s.n_valid = b, e, e
        rc = _lib.device_lib().psdev_dense_op_segs(
            C.byref(t._world), C.byref(t._table), _lib.OP_PUSHPULL, segs, len(ranges),
            C.byref(t._opt_struct()), 0, 0, torch.cuda.current_stream().cuda_stream)
        assert (rc == 0) == ok, (ranges, rc)
    heap.close()


@pytest.mark.parametrize("batch_bytes", [0, 1, 1 << 16, 1 << 22])   # 0: the hooks in Python
def test_rate_changed_between_backward_and_step(cuda_device, batch_bytes):
    """What is still pending goes out with the parameters of the moment: all of a model smaller than
    a batch, or what follows the last launch of a larger one."""
    params = [torch.nn.Parameter(torch.zeros(s, device=cuda_device)) for s in ((8,), (30_000,), (9,))]
    heap, dopt = _optimizer(cuda_device, params, torch.float32, True, batch_bytes)
    for step in range(2):
        dopt.table.optimizer.lr = 0.5
        before = [p.detach().clone() for p in params]
        sum((p * torch.ones_like(p)).sum() for p in params).backward()
        dopt.table.optimizer.lr = 0.25
        dopt.step()
        moved = [b - p.detach() for b, p in zip(before, params)]
        for m in moved:
            assert torch.all(m == m.flatten()[0]) and m.flatten()[0].item() in (0.5, 0.25)
        if batch_bytes == 1 << 22:
            assert all(m.flatten()[0].item() == 0.25 for m in moved)
        if batch_bytes == 1 << 16:
            # the large tensor fills a batch, whichever comes first; a small one stays behind it
            assert 0.25 in [m.flatten()[0].item() for m in moved]
    dopt.close()
    heap.close()


def test_an_error_while_the_parameters_are_read_ends_the_pass(cuda_device):
    """... and the next pass reads them again instead of going on with the old ones."""
    p = torch.nn.Parameter(torch.zeros(64, device=cuda_device))
    heap, dopt = _optimizer(cuda_device, [p], torch.float32, True, 1)
    good = dopt.table.optimizer
    dopt.table.optimizer = None
    with pytest.raises(Exception):
        (p * torch.ones_like(p)).sum().backward()
        dopt.step()
    dopt.table.optimizer = good
    good.lr = 0.125
    dopt.step()
    assert torch.all(p == -0.125)
    dopt.close()
    heap.close()


@pytest.mark.parametrize("step_on_side", [False, True])
@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("batch_bytes", [1, 1 << 22])
def test_hooks_on_two_streams(cuda_device, batch_bytes, overlap, step_on_side):
    """Gradients accumulate on the stream that was current when the parameter first took part in a
    graph: here the default one and another in turn."""
    shapes = [(65,), (300_007,), (4096,), (90_000,), (3,)]
    params = [torch.nn.Parameter(torch.zeros(s, device=cuda_device)) for s in shapes]
    side = torch.cuda.Stream(cuda_device)
    with torch.cuda.stream(side):
        nodes = [p.view_as(p).grad_fn.next_functions[0][0] for p in params[1::2]]
    heap, dopt = _optimizer(cuda_device, params, torch.float32, overlap, batch_bytes)
    assert len(nodes) == 2
    where = []
    for p in params:
        p.register_post_accumulate_grad_hook(
            lambda q: where.append(torch.cuda.current_stream(cuda_device) == side))
    ws = torch.zeros(max(p.numel() for p in params), device=cuda_device)
    for step in range(4):
        for value in (2.0, 4.0):
            x = torch.ones(1, device=cuda_device, requires_grad=True)
            for i, p in enumerate(params):
                x = _FromWorkspace.apply(x, p, value * (i + 1), ws) if i == 0 else x
            (x.sum() + sum((p * torch.full_like(p, value * (i + 1))).sum()
                           for i, p in enumerate(params) if i)).backward()
        if step_on_side:
            side.wait_stream(torch.cuda.current_stream(cuda_device))
            with torch.cuda.stream(side):
                dopt.step()
            torch.cuda.current_stream(cuda_device).wait_stream(side)
        else:
            dopt.step()
        for i, p in enumerate(params):
            assert torch.all(p == -3.0 * (step + 1) * (i + 1)), (step, i)
    assert any(where) and not all(where)
    dopt.close()
    heap.close()


def test_accumulation_stays_on_the_stream_of_the_forward_pass(cuda_device):
    params = [torch.nn.Parameter(torch.zeros(40, device=cuda_device)) for _ in range(2)]
    heap, dopt = _optimizer(cuda_device, params, torch.float32)
    side, where = torch.cuda.Stream(cuda_device), []
    params[0].register_post_accumulate_grad_hook(
        lambda p: where.append(torch.cuda.current_stream(cuda_device) == side))
    for step in range(4):
        side.wait_stream(torch.cuda.current_stream(cuda_device))
        with torch.cuda.stream(side if step % 2 else torch.cuda.current_stream(cuda_device)):
            sum((p * torch.ones_like(p)).sum() for p in params).backward()
            dopt.step()
        torch.cuda.current_stream(cuda_device).wait_stream(side)
    assert where == [False, True, False, True]
    assert all(torch.all(p == -2.0) for p in params)
    dopt.close()
    heap.close()


@pytest.mark.parametrize("overlap", [False, True])
@pytest.mark.parametrize("batch_bytes", [1, 1 << 22])
def test_a_captured_step(cuda_device, batch_bytes, overlap):
    """Forward, backward and update in a CUDA graph, by an optimizer made outside of it."""
    params = [torch.nn.Parameter(torch.zeros(s, device=cuda_device)) for s in ((300, 40), (7,), (90_001,))]
    heap, dopt = _optimizer(cuda_device, params, torch.float32, overlap, batch_bytes)
    coef = [torch.ones_like(p) for p in params]
    ws = torch.zeros(7, device=cuda_device)

    def step():
        x = _FromWorkspace.apply(torch.ones(1, device=cuda_device, requires_grad=True), params[1], 1.0, ws)
        (x.sum() + (params[0] * coef[0]).sum() + (params[2] * coef[2]).sum()).backward()
        dopt.step()

    side = torch.cuda.Stream(cuda_device)
    side.wait_stream(torch.cuda.current_stream(cuda_device))
    with torch.cuda.stream(side):
        for _ in range(2):
            step()
    torch.cuda.current_stream(cuda_device).wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    for n in range(3, 8):
        graph.replay()
        assert all(torch.all(p == -0.5 * n) for p in params), n
    step()
    assert all(torch.all(p == -4.0) for p in params)
    del graph
    dopt.close()
    heap.close()


def test_closed_between_backward_and_step(cuda_device):
    """Gradients whose update has been launched and not waited for keep their memory."""
    n = 1 << 20
    p = torch.nn.Parameter(torch.zeros(n, device=cuda_device))
    heap, dopt = _optimizer(cuda_device, [p], torch.float32, batch_bytes=1)
    at = []
    p.register_hook(lambda g: at.append(g.data_ptr()))
    x = torch.full((n,), 2.0, device=cuda_device)
    torch.cuda.synchronize()
    with torch.cuda.stream(dopt.comm):
        torch.cuda._sleep(400_000_000)   # the update comes behind this: some 0.2 s
    (p * x).sum().backward()
    assert dopt._native.launches == 1 and dopt._native.staged == 0
    dopt._native.detach()
    again = [torch.full((n,), 8.0, device=cuda_device) for _ in range(8)]
    assert at[0] not in [t.data_ptr() for t in again]
    dopt.close()
    assert torch.all(dopt.table.weight[:n] == -1.0)
    heap.close()


@pytest.mark.parametrize("where", ["before", "after", "both"])
def test_tensor_hooks_of_the_program(cuda_device, where):
    """Hooks on the parameters, made before or after the optimizer, see and change the gradients."""
    p, q = (torch.nn.Parameter(torch.zeros(300, device=cuda_device)) for _ in range(2))
    seen = []

    def hook(g):
        seen.append(float(g[0]))
        return 2 * g
    first = p.register_hook(hook) if where != "after" else None
    heap, dopt = _optimizer(cuda_device, [p, q], torch.float32)
    second = p.register_hook(hook) if where != "before" else None
    for _ in range(2):
        (p.sum() + q.sum()).backward()
        dopt.step()
    times = 2 if where == "both" else 1
    assert seen == [1.0, 2.0][:times] * 2
    assert torch.all(p == -2.0 ** times) and torch.all(q == -1.0)
    (second or first).remove()
    (p.sum() + q.sum()).backward()
    dopt.step()
    assert torch.all(p == -2.0 ** times - 2.0 ** (times - 1) / 2) and torch.all(q == -1.5)
    dopt.close()
    if first and second:
        first.remove()
    (p.sum() + q.sum()).backward()
    assert torch.all(p.grad == 1.0) and torch.all(q.grad == 1.0)
    heap.close()
