"""Performance cases of the framework on one GPU.

Each case is one piece of work that a program has the framework do through its public entry
points: requests on dense tensors through :class:`KVStore`, the server-side update of a whole
model through :class:`DistributedOptimizer`, keyed (sparse) steps, the preparation of raw ids
for a push, compressed gradients, and the pull fused with the GEMM that consumes the weights.

``listed()`` names the cases, ``draw(rng)`` gives one more from the same ranges, ``prepare``
makes what the program has in hand before the call, ``run`` makes the call once, ``work`` says
which bytes and operations it cannot do without, ``tolerance`` how far two correct
implementations of the same precision may differ.
"""
import math
import os
import random

import torch

# the libraries are built before anything is measured
os.environ.setdefault("PSB200_NO_BUILD", "1")

from ps_lite_b200 import kvstore  # noqa: E402
from ps_lite_b200.models.bert import BertLarge  # noqa: E402
from ps_lite_b200.models.resnet import ResNet50  # noqa: E402
from ps_lite_b200.ops.gemm import linear_bf16, pull_linear_bf16  # noqa: E402
from ps_lite_b200.ops.keys import sort_unique_sum  # noqa: E402
from ps_lite_b200.parallel import (DenseTable, ServerOptimizer, SparseTable,  # noqa: E402
                                   SymmetricHeap)
from ps_lite_b200.parallel.optimizer import DistributedOptimizer  # noqa: E402

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "int8": torch.int8}
SIZES = {"fp32": 4, "bf16": 2, "int8": 1}
STATES = {"sum": 0, "sgd": 0, "momentum": 1, "adam": 2}
ZIPF = 1.1              # exponent of the id distribution of the sparse workload
ARENA_BYTES = 24 << 30  # of the process-wide job that the KVStore and KeyedStore cases share
WINDOW = 1 << 20        # ids of one keyed state inside its table
WINDOWS = 64
KEYED_MAX = 1 << 17     # keys of one request on a keyed table


# ---- the cases -----------------------------------------------------------------------------------
def listed():
    return [
        # The smallest request: one 4 KiB tensor pushed, updated and pulled (a bias, a batch-norm
        # scale; the lower end of the push/pull sweep).  Latency of the whole request path.
        {"name": "kv_4KiB", "path": "kv", "op": "push_pull", "where": "device", "n": 1024,
         "grad": "fp32", "out": "fp32", "opt": "sgd"},
        # An ordinary layer with an odd number of values, as two requests: gradients pushed after
        # the backward pass, weights pulled before the next forward pass.  bf16 on the wire.
        {"name": "kv_3M_bf16_push_then_pull", "path": "kv", "op": "push_then_pull",
         "where": "device", "n": 3_000_003, "grad": "bf16", "out": "bf16", "opt": "momentum"},
        # The headline point: 256 MiB of fp32 pushed and pulled, SGD on the server, values in the
        # tensor's own buffers.
        {"name": "kv_256MiB_arena", "path": "kv", "op": "push_pull", "where": "arena",
         "n": 64 << 20, "grad": "fp32", "out": "fp32", "opt": "sgd"},
        # The same from pinned host memory and back (a worker whose values live on the host).
        {"name": "kv_64MiB_host", "path": "kv", "op": "push_pull", "where": "host",
         "n": 16 << 20, "grad": "fp32", "out": "fp32", "opt": "sgd"},
        # One update of ResNet-50 (161 tensors, fp32 weights, bf16 gradients, momentum SGD):
        # gradients pushed from the backward hooks, weights pulled in place.
        {"name": "train_resnet50", "path": "train", "model": "resnet50", "opt": "momentum",
         "weights": "fp32"},
        # One update of BERT-large (bf16 weights, server-side Adam on fp32 masters).
        {"name": "train_bert_large", "path": "train", "model": "bert", "opt": "adam",
         "weights": "bf16"},
        # One step of sparse logistic regression: 2^20 Zipf keys of 2^30, FTRL on the server.
        {"name": "sparse_ftrl_2^20", "path": "sparse", "store": "direct", "kind": "ftrl",
         "keys": 1 << 20, "log2_space": 30},
        # A batch of embedding rows (16 values each) pushed and pulled through KVWorker.
        {"name": "keyed_rows_w16", "path": "keyed", "keys": 50_001, "width": 16,
         "var_len": False},
        # Values of different lengths: a push that names them, then a pull that asks for them.
        {"name": "keyed_var_len", "path": "keyed", "keys": 4_099, "width": 8, "var_len": True},
        # The raw ids of a batch, repeats and all, made into the sorted unique keys of a push.
        {"name": "ids_2^22_to_push", "path": "ids", "n": 1 << 22, "bits": 30},
        # A gradient compressed to int8 with one scale per 256 values and pushed in that form.
        {"name": "int8_push_25M", "path": "int8", "n": 25_557_032, "out": "bf16"},
        # The QKV projection of BERT-large (32 x 512 tokens): push of its weight gradient, then
        # the pull fused with the GEMM that consumes the weight.
        {"name": "pull_gemm_qkv", "path": "gemm", "pull": True, "m": 16384, "n": 3072,
         "k": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    path = rng.choices(["kv", "train", "sparse", "keyed", "ids", "int8", "gemm"],
                       [4, 2, 2, 2, 1, 1, 2])[0]
    if path == "kv":
        where = rng.choice(["device", "device", "arena", "host"])
        n = _log(rng, 1 << 10, 64 << 20) if where != "host" else _log(rng, 1 << 14, 16 << 20)
        grad, out = rng.choice([("fp32", "fp32"), ("bf16", "bf16"), ("bf16", "fp32")])
        return {"path": "kv", "op": rng.choice(["push_pull", "push_pull", "push_then_pull"]),
                "where": where, "n": n, "grad": grad, "out": out,
                "opt": rng.choice(["sum", "sgd", "momentum"])}
    if path == "train":
        weights = rng.choice(["fp32", "bf16"])
        return {"path": "train", "model": "mixed", "tensors": _log(rng, 8, 300),
                "total": _log(rng, 1 << 20, 1 << 27), "opt": rng.choice(["momentum", "adam"]),
                "weights": weights}
    if path == "sparse":
        store = rng.choice(["direct", "direct", "hash"])
        return {"path": "sparse", "store": store, "kind": rng.choice(["ftrl", "ftrl", "sgd"]),
                "keys": _log(rng, 1 << 9, 1 << 20),
                "log2_space": rng.randint(24, 30) if store == "direct" else rng.randint(34, 48)}
    if path == "keyed":
        var_len = rng.random() < 0.4
        return {"path": "keyed", "keys": _log(rng, 256, KEYED_MAX),
                "width": 8 if var_len else rng.choice([1, 8, 16]), "var_len": var_len}
    if path == "ids":
        return {"path": "ids", "n": _log(rng, 1 << 12, 1 << 22), "bits": rng.choice([24, 30, 40])}
    if path == "int8":
        return {"path": "int8", "n": _log(rng, 1 << 12, 1 << 26),
                "out": rng.choice(["fp32", "bf16"])}
    return {"path": "gemm", "pull": rng.random() < 0.5, "m": _log(rng, 64, 16384),
            "n": 8 * _log(rng, 32, 512), "k": 8 * _log(rng, 32, 512)}


# ---- inputs --------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _randn(n, g, scale=1.0):
    return torch.randn(n, generator=g, device=g.device).mul_(scale)


def _ranks(n, space, g):
    """``n`` ids with P(rank r) ~ r^-1.1, ranks spread over the key space."""
    u = torch.rand(n, generator=g, device=g.device, dtype=torch.float64).clamp_(1e-300, 1.0)
    r = torch.floor(u.pow(-1.0 / (ZIPF - 1.0))).clamp_(1, space).to(torch.int64) - 1
    return (r * 2654435761) % space


def _unique_zipf(n, space, g):
    """``n`` sorted unique Zipf ids (the request of one worker and step)."""
    keys = torch.empty(0, dtype=torch.int64, device=g.device)
    while keys.numel() < n:
        keys = torch.unique(torch.cat([keys, _ranks(4 * n, space, g)]))
    pick = torch.randperm(keys.numel(), generator=g, device=g.device)[:n]
    return torch.sort(keys[pick]).values


# ---- the job that KVStore and KeyedStore requests belong to --------------------------------------
class _Job:
    """Tensors and tables of a job live as long as the job; a state borrows one and hands it back."""
    store = None
    next_key = 0
    free = {}
    keyed = {}

    @classmethod
    def context(cls):
        if cls.store is None:
            cls.store = kvstore.KVStore(kvstore.init(heap_bytes=ARENA_BYTES))
        return cls.store.ctx


class _Tensor:
    """A declared tensor of the job, on loan."""

    def __init__(self, n, grad, out, opt):
        _Job.context()
        self.config = (n, grad, out, opt)
        idle = _Job.free.setdefault(self.config, [])
        if idle:
            self.key, self.table = idle.pop()
        else:
            self.key = _Job.next_key
            _Job.next_key += 1
            self.table = _Job.store.declare(self.key, n, grad_dtype=DTYPES[grad],
                                            out_dtype=DTYPES[out],
                                            optimizer=ServerOptimizer(opt, lr=0.01))

    def __del__(self):
        _Job.free[self.config].append((self.key, self.table))


class _Heap(SymmetricHeap):
    """A heap of its own, given back when the state and every tensor inside it are gone."""

    def __init__(self, nbytes):
        super().__init__(nbytes + (16 << 20), 0, 1, device=_device())

    def __del__(self):
        self.close()


def _keyed_store(width, var_len):
    """The keyed table of this shape and the first id of a region that no state has used yet."""
    ctx = _Job.context()
    if (width, var_len) not in _Job.keyed:
        app = 1 + len(_Job.keyed)
        _Job.keyed[width, var_len] = [kvstore.KeyedStore(
            ctx, app, WINDOW * WINDOWS, KEYED_MAX, width=width, kind="sgd", lr=0.05,
            var_len=var_len), 0]
    entry = _Job.keyed[width, var_len]
    first = entry[1] % WINDOWS * WINDOW
    entry[1] += 1
    return entry[0], first


# ---- dense requests ------------------------------------------------------------------------------
def _prepare_kv(case, seed):
    g, n = _generator(seed), case["n"]
    lent = _Tensor(n, case["grad"], case["out"], case["opt"])
    t = lent.table
    t.load_master(_randn(n, g, 0.05))
    if t.state1 is not None:
        t.state1.zero_()
    grad = _randn(n, g).to(DTYPES[case["grad"]])
    value = out = None
    if case["where"] == "device":
        value, out = grad, torch.empty(n, dtype=DTYPES[case["out"]], device=g.device)
    elif case["where"] == "host":
        value = torch.empty(n, dtype=grad.dtype, pin_memory=True).copy_(grad)
        out = torch.empty(n, dtype=DTYPES[case["out"]], pin_memory=True)
    else:
        t.grad[:n].copy_(grad)
    return {"store": _Job.store, "lent": lent, "value": value, "out": out, "n": n}


def _run_kv(case, s):
    kv, key, t = s["store"], s["lent"].key, s["lent"].table
    if case["op"] == "push_pull":
        kv.wait(kv.push_pull(key, s["value"], s["out"]))
    else:
        kv.wait(kv.push(key, s["value"]))
        kv.wait(kv.pull(key, s["out"]))
    return {"pulled": t.weight[: s["n"]] if s["out"] is None else s["out"], "master": t.master,
            "state": t.state1}


# ---- one update of a model -----------------------------------------------------------------------
def _shapes(case):
    if case["model"] != "mixed":
        with torch.device("meta"):
            model = ResNet50() if case["model"] == "resnet50" else BertLarge()
        return [tuple(p.shape) for p in model.parameters()]
    rng = random.Random(case["tensors"] * 1_000_003 + case["total"])
    parts = [math.exp(rng.gauss(0.0, 2.0)) for _ in range(case["tensors"])]
    return [(max(1, int(case["total"] * p / sum(parts))),) for p in parts]


class _Backward(torch.autograd.Function):
    """A backward pass that hands over ready gradients: the exchange without a model's kernels."""

    @staticmethod
    def forward(ctx, grads, *params):
        ctx.grads = grads
        return params[0].new_zeros(())

    @staticmethod
    def backward(ctx, _):
        return (None, *[g.view(g.shape) for g in ctx.grads])


class _Trainer:
    """The optimizer of a model, detached from its parameters with the state."""

    def __init__(self, params, heap, opt):
        self.dopt = DistributedOptimizer(params, heap, opt, grad_dtype=torch.bfloat16)

    def __del__(self):
        self.dopt.close()


def _prepare_train(case, seed):
    g, dtype, shapes = _generator(seed), DTYPES[case["weights"]], _shapes(case)
    total = sum((math.prod(s) + 7) // 8 * 8 for s in shapes)
    own = _Heap(total * (2 + SIZES[case["weights"]]) + (1 << 20))
    weights = _randn(total, g, 0.05).to(dtype)
    grads = _randn(total, g).to(dtype)
    params, gs, at = [], [], 0
    for s in shapes:
        k = math.prod(s)
        params.append(torch.nn.Parameter(weights[at:at + k].view(s)))
        gs.append(grads[at:at + k].view(s))
        at += (k + 7) // 8 * 8
    opt = ServerOptimizer(case["opt"], lr=0.01, momentum=0.9) if case["opt"] == "momentum" else \
        ServerOptimizer("adam", lr=1e-4, eps=1e-6)
    return {"params": params, "grads": gs, "trainer": _Trainer(params, own, opt)}


def _run_train(case, s):
    dopt = s["trainer"].dopt
    dopt.zero_grad()
    _Backward.apply(s["grads"], *s["params"]).backward()
    dopt.step()
    t = dopt.table
    return {"weight": t.weight, "master": t.master, "state1": t.state1, "state2": t.state2}


# ---- keyed tables --------------------------------------------------------------------------------
def _prepare_sparse(case, seed):
    g, n, space = _generator(seed), case["keys"], 1 << case["log2_space"]
    capacity = 4 * (1 << (n - 1).bit_length()) if case["store"] == "hash" else 0
    slots = capacity or space
    own = _Heap(4 * slots + 8 * capacity + 16 * n)
    table = SparseTable(own, space, n, kind=case["kind"], hash_capacity=capacity)
    return {"table": table, "keys": _unique_zipf(n, space, g),
            "grads": _randn(n, g, 2.0)}


def _run_sparse(case, s):
    t = s["table"]
    values = t.push_pull(s["keys"], s["grads"])
    if case["store"] == "hash":  # which slot a key gets depends on the order of arrival
        return {"values": values}
    return {"values": values, "w": t.w, "z": t.z, "n": t.n}


def _packed(n, width):
    """Values of ``n`` keys whose lengths are spread evenly over 1..width."""
    return n // width * (width * (width + 1) // 2) + n % width * (n % width + 1) // 2


def _prepare_keyed(case, seed):
    g, n, width = _generator(seed), case["keys"], case["width"]
    store, first = _keyed_store(width, case["var_len"])
    keys = _unique_zipf(n, WINDOW, g) + first
    s = {"store": store, "keys": keys, "lens": None, "lens_out": None}
    count = n * width
    if case["var_len"]:
        order = torch.randperm(n, generator=g, device=g.device)
        s["lens"] = (order % width + 1).to(torch.int32)
        s["lens_out"] = torch.empty_like(s["lens"])
        count = _packed(n, width)
    s["vals"] = _randn(count, g)
    s["out"] = torch.empty_like(s["vals"])
    return s


def _run_keyed(case, s):
    store = s["store"]
    if case["var_len"]:
        store.wait(store.push(s["keys"], s["vals"], s["lens"]))
        store.wait(store.pull(s["keys"], s["out"], s["lens_out"]))
        return {"out": s["out"], "lens": s["lens_out"]}
    store.wait(store.push_pull(s["keys"], s["vals"], s["out"]))
    return {"out": s["out"]}


# ---- the rest ------------------------------------------------------------------------------------
def _prepare_ids(case, seed):
    # as many different ids as Zipf draws have, each at least once, the popular ones often
    g, n, u = _generator(seed), case["n"], _distinct(case["n"], case["bits"])
    known = _unique_zipf(u, 1 << case["bits"], g)
    ids = torch.cat([known, known[_ranks(n - u, u, g)]])
    return {"ids": ids[torch.randperm(n, generator=g, device=g.device)], "vals": _randn(n, g)}


def _run_ids(case, s):
    keys, sums = sort_unique_sum(s["ids"], s["vals"], key_bits=case["bits"])
    return {"keys": keys, "sums": sums}


def _prepare_int8(case, seed):
    g, n = _generator(seed), case["n"]
    own = _Heap(n * (1 + SIZES[case["out"]]) + n // 64 + (1 << 20))
    t = DenseTable(own, n, torch.int8, DTYPES[case["out"]],
                   optimizer=ServerOptimizer("momentum", lr=0.01))
    t.load_master(_randn(n, g, 0.05))
    return {"table": t, "grad": _randn(n, g)}


def _run_int8(case, s):
    t = s["table"]
    t.stage_int8(s["grad"])
    t.push_pull()
    return {"codes": t.grad, "scales": t.gscale, "weight": t.weight, "master": t.master,
            "state": t.state1}


def _prepare_gemm(case, seed):
    g, m, n, k = _generator(seed), case["m"], case["n"], case["k"]
    s = {"x": _randn(m * k, g).to(torch.bfloat16).view(m, k)}
    w = _randn(n * k, g, k ** -0.5)
    if case["pull"]:
        s["table"] = DenseTable(_Heap(4 * n * k + (1 << 20)), n * k, torch.bfloat16, torch.bfloat16, blk=4096,
                                optimizer=ServerOptimizer("sgd", lr=0.01))
        s["table"].load_master(w)
        s["table"].grad.copy_(_randn(n * k, g))
    else:
        s["w"] = w.to(torch.bfloat16).view(n, k)
    return s


def _run_gemm(case, s):
    if not case["pull"]:
        return {"out": linear_bf16(s["x"], s["w"])}
    t = s["table"]
    t.push(publish=True)
    out = pull_linear_bf16(t, 0, case["n"], s["x"])
    return {"out": out, "weight": t.weight, "master": t.master}


_PREPARE = {"kv": _prepare_kv, "train": _prepare_train, "sparse": _prepare_sparse,
            "keyed": _prepare_keyed, "ids": _prepare_ids, "int8": _prepare_int8,
            "gemm": _prepare_gemm}
_RUN = {"kv": _run_kv, "train": _run_train, "sparse": _run_sparse, "keyed": _run_keyed,
        "ids": _run_ids, "int8": _run_int8, "gemm": _run_gemm}


def prepare(case, seed):
    state = _PREPARE[case["path"]](case, seed)
    state["case"] = case
    return state


def run(state):
    case = state["case"]
    return _RUN[case["path"]](case, state)


# ---- what a pass cannot do without ---------------------------------------------------------------
def _distinct(n, bits):
    """Expected number of different ids among ``n`` Zipf draws, octave by octave."""
    total, tail = 0.0, ZIPF - 1.0
    for b in range(bits):
        p = 2.0 ** (-tail * b) - 2.0 ** (-tail * (b + 1))
        total += 2.0 ** b * -math.expm1(-n * p / 2.0 ** b)
    return int(total)


def work(case):
    path = case["path"]
    if path == "kv":
        # gradient in, fp32 master and state read and written, new weights out; from the host the
        # same bytes also cross PCIe, which bounds that form
        n = case["n"]
        return {"bytes": n * (SIZES[case["grad"]] + SIZES[case["out"]] + 8 +
                              8 * STATES[case["opt"]]), "flops": 2 * n}
    if path == "train":
        n, w = sum(math.prod(s) for s in _shapes(case)), SIZES[case["weights"]]
        return {"bytes": n * (2 * w + 8 + 8 * STATES[case["opt"]]), "flops": 8 * n}
    if path == "sparse":
        n = case["keys"]
        return {"bytes": n * (16 + (24 if case["kind"] == "ftrl" else 8)), "flops": 10 * n}
    if path == "keyed":
        n = case["keys"]
        vals = _packed(n, case["width"]) if case["var_len"] else n * case["width"]
        # (the lengths are named by the push and returned by the pull, and the owner keeps them)
        return {"bytes": 8 * n + 16 * vals + (16 * n if case["var_len"] else 0), "flops": 2 * vals}
    if path == "ids":
        return {"bytes": 12 * case["n"] + 12 * _distinct(case["n"], case["bits"]),
                "flops": case["n"]}
    if path == "int8":
        # gradient in, codes and scales out, master and momentum read and written, weights out
        n = case["n"]
        return {"bytes": n * (4 + 1 + 16 + SIZES[case["out"]]) + n // 64, "flops": 8 * n}
    m, n, k = case["m"], case["n"], case["k"]
    moved = 2 * (m * k + n * k + m * n)
    if case["pull"]:
        moved += n * k * (2 + 8)
    return {"bytes": moved, "flops": 2 * m * n * k}


def tolerance(case):
    path = case["path"]
    if path == "gemm":
        # bf16 results of fp32 accumulation: half a unit in the last place is 2^-9
        return {"rel": 4e-3, "max": 3e-2}
    if "bf16" in (case.get("out"), case.get("weights")):
        # fp32 updates; a weight next to a rounding boundary may fall to the other side in bf16
        return {"rel": 1e-3, "max": 1e-2, "differ": 1e-5}
    if path == "ids":
        # the most popular id of a large batch adds up some 10^5 values, in any order
        return {"rel": 5e-5, "max": 2e-3}
    return {"rel": 1e-5, "max": 1e-3, "differ": 1e-5 if path == "int8" else 0.0}
