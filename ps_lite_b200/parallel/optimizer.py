"""Data-parallel training through the parameter server: gradients are pushed as they are
produced, the server-side optimizer runs on the owners, weights are pulled before the next
forward pass.

The pattern is the one the reference documents for synchronous SGD (docs/overview.md:79-122)
and that its users build on ``KVWorker::Push/Pull`` with per-message priorities
(include/ps/kv_app.h:114-123; priority send queue, src/p3_van.h:12-57).  Here

* all parameters live in one :class:`DenseTable`; a parameter's storage *is* its slice of the
  pulled-weight buffer, so a pull updates the model in place;
* a gradient hook copies (and casts) each gradient into the table's gradient buffer and hands
  its slices to a priority scheduler; slices are at most ``slice_bytes`` long (4 MB by
  default) and their priority is the reverse of the layer order, so the weights the next
  forward pass needs first are exchanged first among the slices that are pending;
* on one rank there is nothing to exchange: native hooks (src/torch/grad_exchange.cc) collect the
  gradient tensors as they are, and the update kernel reads them where they lie; a gradient whose
  memory somebody else can still write (a view of a workspace, say) is copied by its hook;
* slices are exchanged by fused push+pull kernels on a side stream, overlapping the rest of
  backward: as soon as ``batch_bytes`` (4 MiB by default, on one rank a quarter of the model, 4 to
  32; ``PSB200_BATCH_BYTES``) are pending, everything pending goes out in ONE launch whose CTAs take
  the slices in priority order, so small tensors share a rendezvous (on one rank up to four batches
  wait while the launch before is still running); with ``batch_bytes=0`` every hook launches up to
  ``slices_per_event`` single-slice kernels and the rest waits in the host queue.

Every rank makes the same scheduling decisions because they depend only on the order in which
gradient hooks fire, which is the same on every rank for the same model.
"""
from __future__ import annotations

import ctypes as C
import heapq
import weakref
from typing import Iterable, List, Optional, Tuple

import torch

from .. import _lib
from .dense import DenseTable, ServerOptimizer
from .heap import SymmetricHeap


# Bytes of gradients that a launch waits for, unless the program says otherwise.  Several ranks, and
# the hooks in Python: enough that small tensors share a rendezvous.
BATCH_BYTES = 4 << 20
# The native hooks of one rank have no rendezvous, but every launch costs their thread some 5 us
# (300 tensors with 2^27 values, ready gradients: 3777 us with 34 launches, 3635 with 7; the 297 tensors
# of BERT-large 3763 with 37, 3605 with 19).  A quarter of the model within these bounds, so that the
# rest is updated beside the backward pass ...
BATCH_ONE_RANK = 4 << 20, 32 << 20
# ... and more while the launch before is still running: what is sent would only queue up behind it
# and take SMs from the backward pass.  (A program that names its batch: four of them.  Three layers of
# 2048 x 2048, 16384 rows, Adam, batches of 4 MiB: 1488 us, 1548 when none waits.)
BATCH_BUSY = 16 << 20


class P3Scheduler:
    """Priority queue of (begin, end) slices of one table; highest priority first, FIFO among
    equal priorities (same order as ``ThreadsafePQueue`` of the host runtime)."""

    def __init__(self, slice_elems: int):
        self.slice_elems = max(8, int(slice_elems) & ~7)
        self._heap: List[Tuple[int, int, int, int]] = []
        self._seq = 0
        self.pending_elems = 0

    def add(self, begin: int, end: int, priority: int) -> int:
        """Cut [begin, end) into slices and queue them; returns the number of slices."""
        n = 0
        b = begin
        while b < end:
            e = min(b + self.slice_elems, end)
            heapq.heappush(self._heap, (-priority, self._seq, b, e))
            self.pending_elems += e - b
            self._seq += 1
            n += 1
            b = e
        return n

    def pop(self) -> Optional[Tuple[int, int, int]]:
        if not self._heap:
            return None
        negp, _, b, e = heapq.heappop(self._heap)
        self.pending_elems -= e - b
        return b, e, -negp

    def __len__(self) -> int:
        return len(self._heap)


class DistributedOptimizer:
    """Server-side optimizer for the parameters of a model, one process per GPU."""

    def __init__(self, params: Iterable[torch.nn.Parameter], heap: SymmetricHeap,
                 optimizer: ServerOptimizer, grad_dtype=torch.bfloat16, blk: int = 4096,
                 slice_bytes: int = 4 << 20, slices_per_event: int = 2, channel: int = 0,
                 num_ctas: int = 32, overlap: bool = True, publish_first: int = 0,
                 nvls: Optional[bool] = None, publish_params=(),
                 batch_bytes: Optional[int] = None):
        self.params = [p for p in params if p.requires_grad]
        if not self.params:
            raise ValueError("no trainable parameters")
        wdt = self.params[0].dtype
        if any(p.dtype != wdt for p in self.params):
            raise ValueError("all parameters must share one dtype")
        self.heap = heap
        self.offsets, off = [], 0
        for p in self.params:
            self.offsets.append(off)
            off += (p.numel() + 7) & ~7
        self.total = off
        self.table = DenseTable(heap, self.total, grad_dtype, wdt, blk=blk, optimizer=optimizer,
                                channel=channel, num_ctas=num_ctas, nvls=nvls)
        gsz = torch.empty((), dtype=grad_dtype).element_size()
        self.sched = P3Scheduler(slice_bytes // gsz)
        self.slices_per_event = slices_per_event
        # gradients wait in the queue until `batch_bytes` are pending, then everything pending
        # goes out in one launch (small tensors share a rendezvous); 0 = launch from every hook
        if batch_bytes is None:
            import os
            batch_bytes = os.environ.get("PSB200_BATCH_BYTES")
        self.batch_bytes = BATCH_BYTES if batch_bytes is None else int(batch_bytes)
        self._busy_bytes = 4 * self.batch_bytes
        if batch_bytes is None and self._native_ok(grad_dtype):
            least, most = BATCH_ONE_RANK
            self.batch_bytes = min(most, max(least, self.total * gsz // 4))
            self._busy_bytes = max(BATCH_BUSY, self.batch_bytes)
        self._gsz = gsz
        self.launches = 0
        self.overlap = overlap
        self.comm = torch.cuda.Stream(heap.device) if overlap else None
        # the first `publish_first` parameters are pushed with publish instead of push+pull:
        # their weights are pulled by a GEMM-fused pull in the next forward pass
        self.publish_first = publish_first
        pub = {id(p) for p in publish_params}
        self._publish = [i < publish_first or id(p) in pub for i, p in enumerate(self.params)]
        self.steps = 0
        self.launched_slices = 0
        # initial weights: rank 0's values, installed through an "assign" push
        full = torch.zeros(self.total, dtype=torch.float32, device=heap.device)
        for p, o in zip(self.params, self.offsets):
            full[o:o + p.numel()] = p.detach().reshape(-1).float()
        heap.broadcast(full, 0)
        self.table.load_master(full)
        self.table.pull()
        torch.cuda.synchronize(heap.device)
        # a parameter's storage is its slice of the pulled-weight buffer
        for p, o in zip(self.params, self.offsets):
            p.data = self.table.weight[o:o + p.numel()].view(p.shape)
        self._hooks, self._native = [], None
        if self._native_ok(grad_dtype):
            self._native = self._make_native(channel, slice_bytes // gsz)
        else:
            self._hooks = [p.register_post_accumulate_grad_hook(self._make_hook(i))
                           for i, p in enumerate(self.params)]
        self._pending_step = False

    def _native_ok(self, grad_dtype) -> bool:
        """One rank, gradients in a type that the update kernel reads in place, and batching on
        (``batch_bytes=0`` asks for a launch per slice)."""
        return (self.heap.world == 1 and not self.heap.emulated_ranks and self.batch_bytes > 0 and
                grad_dtype in (torch.float32, torch.bfloat16) and
                all(p.is_cuda for p in self.params))

    def _make_native(self, channel: int, slice_elems: int):
        t = self.table
        self._opt = opt = _lib.Opt()
        me = weakref.ref(self)   # (the native object must not keep its owner alive)

        def refresh():
            # the handle's parameters as they are at each launch: a program may change the rate
            # between the backward pass and the step
            t.step = me().steps + 1
            C.memmove(C.byref(opt), C.byref(t._opt_struct()), C.sizeof(opt))

        segs, copy = (C.cast(f, C.c_void_p).value for f in (self.heap.lib.psdev_dense_op_segs,
                                                             self.heap.lib.psdev_copy_cast))
        # reverse layer order, published parameters last (on one rank publishing is the same
        # store into this rank's weight buffer)
        pri = [-1 - i if self._publish[i] else len(self.params) - i
               for i in range(len(self.params))]
        # torch drops the native hooks of a tensor when the first hook in Python arrives; once it
        # has had one, later ones are added beside the native one
        for p in self.params:
            if p._backward_hooks is None:
                p.register_hook(lambda g: None).remove()
        # `num_ctas` bounds the CTAs that wait for peers while a backward pass needs the SMs; with
        # one rank the update is a pass over memory, shortest on the whole GPU
        return _lib.torch_ext().GradExchange(
            self.params, self.offsets, pri, t.grad, C.addressof(t._world), C.addressof(t._table),
            C.addressof(self._opt), segs, copy, self.comm.cuda_stream if self.comm else 0,
            self.comm is not None, max(1, self.batch_bytes // self._gsz),
            max(1, self._busy_bytes // self._gsz), max(8, int(slice_elems) & ~7), channel, refresh)

    def _make_hook(self, index: int):
        n_params = len(self.params)

        o = self.offsets[index]
        n = self.params[index].numel()
        # the parameter's slice of the gradient buffer, in the parameter's shape (made once: the
        # hook runs on the autograd thread, between the kernels of the backward pass)
        gview = self.table.grad[o:o + n].view(self.params[index].shape)

        def hook(p: torch.nn.Parameter):
            gview.copy_(p.grad, non_blocking=True)
            p.grad = None
            if not self._pending_step:
                self._pending_step = True
                self.table.step = self.steps + 1
            # reverse layer order: parameter 0 (needed first by the next forward) is most urgent
            pri = n_params - index
            if self._publish[index]:
                pri = -1 - index  # published slices carry no pull: least urgent
            self.sched.add(o, o + ((n + 7) & ~7), pri)
            if self.batch_bytes <= 0:
                self._launch(self.slices_per_event)
            elif self.sched.pending_elems * self._gsz >= self.batch_bytes:
                self._drain()
        return hook

    def _launch(self, count: int) -> None:
        if count <= 0 or not len(self.sched):
            return
        cur = torch.cuda.current_stream(self.heap.device)
        stream = self.comm or cur
        if self.comm is not None:
            self.comm.wait_stream(cur)
        for _ in range(count):
            item = self.sched.pop()
            if item is None:
                break
            b, e, pri = item
            if pri < 0:
                self.table.push(b, e, stream=stream, opt_step=False, publish=True)
            else:
                self.table.push_pull(b, e, stream=stream, opt_step=False)
            self.launched_slices += 1
            self.launches += 1

    def _drain(self) -> None:
        """Everything queued goes out in one launch per kind of operation; the kernel itself
        takes the slices in priority order (device-side schedule)."""
        if not len(self.sched):
            return
        cur = torch.cuda.current_stream(self.heap.device)
        stream = self.comm or cur
        if self.comm is not None:
            self.comm.wait_stream(cur)
        both, publish = [], []
        while True:
            item = self.sched.pop()
            if item is None:
                break
            (publish if item[2] < 0 else both).append(item)
        cap = self.table.MAX_SEGS
        if len(both) == 1:
            b, e, _ = both[0]
            self.table.push_pull(b, e, stream=stream, opt_step=False)
            self.launches += 1
        else:
            for i in range(0, len(both), cap):
                self.table.run_multi(_lib.OP_PUSHPULL, both[i:i + cap], stream=stream)
                self.launches += 1
        for i in range(0, len(publish), cap):
            self.table.run_multi(_lib.OP_PUSH | _lib.OP_PUBLISH, publish[i:i + cap], stream=stream)
            self.launches += 1
        self.launched_slices += len(both) + len(publish)

    def step(self) -> None:
        """Finish the exchange of this step's gradients; afterwards the parameters hold the
        weights for the next forward pass (except published ones, which their GEMM pulls)."""
        if self._native is not None:
            self._native.step()
            self.launches, self.launched_slices = self._native.launches, self._native.slices
            self.steps += 1
            return
        self._drain()
        if self.comm is not None:
            torch.cuda.current_stream(self.heap.device).wait_stream(self.comm)
        self.steps += 1
        self._pending_step = False

    def zero_grad(self) -> None:
        for p in self.params:
            p.grad = None

    def check(self) -> None:
        self.table.check()

    def close(self) -> None:
        """Detach from the model and give the table's buffers back to the heap.  The
        parameters keep pointing at the pulled-weight buffer: drop the model too."""
        for h in self._hooks:
            h.remove()
        self._hooks = []
        if self._native is not None:
            self._native.detach()
            self._native = None
        torch.cuda.synchronize(self.heap.device)
        self.table.free()

    def offset_of(self, param: torch.nn.Parameter) -> int:
        for p, o in zip(self.params, self.offsets):
            if p is param:
                return o
        raise KeyError("parameter not managed by this optimizer")
