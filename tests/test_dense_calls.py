"""What DenseTable hands to the library, with stand-ins for the library and the streams (no GPU)."""
import ctypes as C
import gc
import types
import weakref

import pytest
import torch

from ps_lite_b200 import _lib
from ps_lite_b200.parallel.dense import DenseTable, ServerOptimizer


@pytest.fixture
def table(monkeypatch):
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: 7, raising=False)
    t = object.__new__(DenseTable)
    t.optimizer, t.step, t.n, t.nvls = ServerOptimizer("adam", lr=0.5), 0, 1024, False
    t._opt_key, t._opt_cached, t._opt_step, t._opt_at = None, None, -1, 0
    t._default_timeout, t.grad_size, t._device_index = 1.0, 1, 0
    t.channel = t.num_ctas = t._op_fn = t._world_at = t._table_at = 0
    t.calls = []

    def op(*args):
        t.calls.append(_lib.Opt.from_buffer_copy(_lib.Opt.from_address(args[6])))
        return 0
    t._dense_op = op
    return t


def test_parameters_live_as_long_as_the_call(table):
    """Another thread that changes the rate during the call replaces the structure."""
    def op(*args):
        at = weakref.ref(table._opt_cached)
        assert args[6] == C.addressof(at())
        table.optimizer.lr = 0.25
        table._opt_struct()
        gc.collect()
        assert at() is not None and _lib.Opt.from_address(args[6]).lr == 0.5
        return 0
    table._dense_op = op
    table.push()


def test_parameters_that_a_class_of_the_program_computes(table):
    class Warmup(ServerOptimizer):
        rate = 1.0
        lr = property(lambda self: self.rate, lambda self, value: None)
    table.optimizer = Warmup("sgd")
    table.push()
    Warmup.rate = 0.125
    table.push()
    table.push()
    assert [o.lr for o in table.calls] == [1.0, 0.125, 0.125]


def test_parameters_follow_the_fields_and_the_step(table):
    table.push()
    table.push_pull()
    table.optimizer.lr = 0.25
    table.pull()
    table.optimizer = ServerOptimizer("sgd", lr=2.0)
    table.push()
    assert [o.lr for o in table.calls] == [0.5, 0.5, 0.25, 2.0]
    assert table.calls[0].bias1 != table.calls[1].bias1


def test_a_gradient_counted_from_the_end(table):
    """stage_int8 with a negative begin, as in a slice; beyond the end it is refused."""
    got = []
    table.gscale, table.grad = torch.zeros(4), torch.zeros(1024, dtype=torch.int8)
    table.heap = types.SimpleNamespace(lib=types.SimpleNamespace(
        psdev_filter_int8_pack=lambda src, dst, scale, n, stream: got.append((dst, scale, n)) or 0))
    for begin, n in ((0, 1024), (256, 300), (-256, 256), (-1024, 5), (-1280, 256)):
        table.stage_int8(torch.zeros(n), begin)
        at = max(begin + 1024, 0) if begin < 0 else begin
        assert got[-1] == (table.grad[at:].data_ptr(), table.gscale[at // 256:].data_ptr(), n)
    for begin, n in ((0, 1025), (-256, 257), (-1280, 1025), (1024, 1)):
        with pytest.raises(ValueError):
            table.stage_int8(torch.zeros(n), begin)


def test_streams_are_those_of_the_memory_s_device():
    """A heap may name its device without an index."""
    memory = types.SimpleNamespace(device=types.SimpleNamespace(index=3), zero_=lambda: None)
    op = C.CFUNCTYPE(C.c_int)(lambda: 0)
    heap = types.SimpleNamespace(
        world=1, mc_base=0, emulated_ranks=False, device=torch.device("cpu"),
        alloc=lambda nbytes: 256, tensor=lambda off, n, dtype: memory,
        world_struct=_lib.World, lib=types.SimpleNamespace(psdev_dense_op=op))
    assert DenseTable(heap, 64)._device_index == 3
