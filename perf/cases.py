"""The work that users of this library have it do on one GPU, as timed cases.

Two kinds of communicator serve one GPU, and both are used in earnest:

* ``world = 1``: a process group of one rank over symmetric memory, what a tensor-parallel
  program runs on when it is started on a single GPU.  The collectives degenerate to local
  copies; the GEMMs, the fused operators and the host path are the ones of the larger groups.
* ``world >= 2``: an emulated world, all ranks of a collective in one launch on one GPU, which
  is how programs for more GPUs are developed and tested; the multi-rank kernels run unchanged.

Message sizes follow the size sweep (1 KiB up to the headline 512 MiB), layer sizes the default
of the tensor-parallel MLP block (hidden 4096, intermediate 14336) and what the tests use.
"""
import torch
import torch.distributed as dist

import tccl_b200 as tccl
from tccl_b200.config import Config
from tccl_b200.models import TensorParallelMLP
from tccl_b200.ops.gemm import gemm_bf16
from tccl_b200.ops.quantized import QUANT_CHUNK
from tccl_b200.parallel.emu import EmuWorld

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
SIZE = {"bf16": 2, "fp16": 2, "fp32": 4}
DEVICE = "cuda"


def listed():
    return [
        # the message of one decode step on one rank: all latency
        {"name": "all_reduce 8 KiB, 1 rank", "op": "all_reduce", "world": 1, "dtype": "bf16", "numel": 4096, "out": "new"},
        # the headline message: bandwidth
        {"name": "all_reduce 512 MiB, 1 rank", "op": "all_reduce", "world": 1, "dtype": "bf16", "numel": 1 << 28, "out": "symmetric"},
        # a small activation, summed over eight ranks (tests and decode steps of programs for eight GPUs)
        {"name": "all_reduce 16 KiB, 8 ranks", "op": "all_reduce", "world": 8, "dtype": "bf16", "numel": 8192, "out": "new"},
        # gradients or prefill activations over eight ranks, larger than L2
        {"name": "all_reduce 32 MiB, 8 ranks", "op": "all_reduce", "world": 8, "dtype": "bf16", "numel": 1 << 24, "out": "symmetric"},
        # shards of a parameter tensor whose size is nobody's multiple
        {"name": "all_gather ragged, 4 ranks", "op": "all_gather", "world": 4, "dtype": "fp32", "numel": 1000003, "out": "new"},
        # gradients to their owners
        {"name": "reduce_scatter 32 MiB, 8 ranks", "op": "reduce_scatter", "world": 8, "dtype": "fp16", "numel": 1 << 24, "out": "new"},
        # the double tree, in the range where it is chunked and pipelined
        {"name": "tree 8 MiB, 4 ranks", "op": "tree", "world": 4, "dtype": "fp32", "numel": 1 << 21, "out": "new"},
        # fp8 on the wire
        {"name": "quantized 16 MiB, 8 ranks", "op": "quantized", "world": 8, "dtype": "bf16", "numel": 1 << 23, "out": "new"},
        # a projection of a token count that is no multiple of a tile
        {"name": "gemm 1000x1792x4096", "op": "gemm", "m": 1000, "n": 1792, "k": 4096},
        # prefill of the MLP block in its sequence-parallel form: all-gather -> GEMM + SwiGLU, GEMM -> reduce-scatter
        {"name": "mlp prefill 4096, 1 rank", "op": "mlp", "form": "sequence", "world": 1, "tokens": 4096, "hidden": 4096, "inter": 14336},
        # a decode step of the same block in its all-reduce form: GEMMs of few rows, all-reduce + residual + RMSNorm
        {"name": "mlp decode 16, 1 rank", "op": "mlp", "form": "all_reduce", "world": 1, "tokens": 16, "hidden": 4096, "inter": 14336},
        # the two fused GEMM kernels with four ranks exchanging tiles
        {"name": "mlp prefill 2048, 4 ranks", "op": "mlp", "form": "sequence", "world": 4, "tokens": 2048, "hidden": 2048, "inter": 7168},
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    op = rng.choice(["all_reduce", "all_reduce", "all_gather", "reduce_scatter", "tree", "quantized", "gemm", "mlp", "mlp"])
    if op == "gemm":
        # from one decode row to a prefill; the widths that the operator takes are multiples of 8
        return {"op": op, "m": _log(rng, 1, 4096), "n": 8 * _log(rng, 32, 1792), "k": 8 * _log(rng, 32, 1792)}
    if op == "mlp":
        hidden, inter = rng.choice([(1024, 3584), (2048, 7168), (4096, 14336)])
        if rng.random() < 0.5:
            return {"op": op, "form": "all_reduce", "world": 1, "tokens": _log(rng, 1, 2048), "hidden": hidden, "inter": inter}
        world = rng.choice([1, 1, 2, 4])
        rows = 128 * world  # whole 128-row tiles per rank
        return {"op": op, "form": "sequence", "world": world, "tokens": rows * _log(rng, 1, 4096 // rows), "hidden": hidden, "inter": inter}
    world = rng.choice([1, 2, 3, 4, 8])
    dtype = "bf16" if op == "quantized" else rng.choice(["bf16", "fp32", "fp16"])
    nbytes = _log(rng, 1 << 10, (256 << 20) // world)  # per rank
    numel = nbytes // SIZE[dtype]
    if op == "quantized":
        numel = max(1, numel // QUANT_CHUNK) * QUANT_CHUNK
    elif op == "reduce_scatter":
        unit = 16 // SIZE[dtype] * world  # the operator's own rule
        numel = max(1, numel // unit) * unit
    elif op == "tree":
        unit = 16 // SIZE[dtype]
        numel = max(1, numel // unit) * unit
    elif op == "all_gather":
        numel = max(1, numel // world)  # the gathered tensor is `world` shards
    out = "symmetric" if op == "all_reduce" and rng.random() < 0.5 else "new"
    return {"op": op, "world": world, "dtype": dtype, "numel": numel, "out": out}


# ------------------------------------------------------------------ communicators, one of each kind per process
_worlds = {}


def _world(size):
    if size not in _worlds:
        if size == 1:
            torch.cuda.set_device(0)
            dist.init_process_group("nccl", store=dist.HashStore(), rank=0, world_size=1, device_id=torch.device("cuda", 0))
            _worlds[1] = tccl.init()
        else:
            _worlds[size] = EmuWorld(size, config=Config.from_env())
    return _worlds[size]


class State:
    """What a program holds between calls; gives its symmetric tensors back when it goes."""

    def __init__(self, world, op):
        self.world, self.op, self.symmetric = world, op, []

    def empty(self, shape, dtype):
        t = self.world.empty(shape, dtype)
        if self.world.world_size == 1:
            self.symmetric.append(t)
        return t

    def __del__(self):
        for t in self.symmetric:
            self.world.free(t)


def _normal(gen, shape, dtype, scale=1.0):
    return (torch.randn(shape, generator=gen, device=DEVICE, dtype=torch.float32) * scale).to(dtype)


def _fill(gen, t):
    """N(0, 1) into one rank's tensor, a block at a time (the largest is 512 MiB)."""
    flat, step = t.view(-1), 1 << 25
    for i in range(0, flat.numel(), step):
        n = min(step, flat.numel() - i)
        flat[i: i + n] = torch.randn(n, generator=gen, device=DEVICE)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    op = case["op"]
    if op == "gemm":
        s = State(None, op)
        s.a = _normal(gen, (case["m"], case["k"]), torch.bfloat16)
        s.bt = _normal(gen, (case["n"], case["k"]), torch.bfloat16, 0.02)
        return s
    w = _world(case["world"])
    s = State(w, op)
    if op == "mlp":
        s.op = "mlp_" + case["form"]
        T, H, F, W = case["tokens"], case["hidden"], case["inter"], case["world"]
        weights = (_normal(gen, (F, H), torch.bfloat16, 0.02), _normal(gen, (F, H), torch.bfloat16, 0.02),
                   _normal(gen, (H, F), torch.bfloat16, 0.02))
        blocks = [TensorParallelMLP(w, r, H, F, device=DEVICE, full_weights=weights) for r in range(W)]
        x = _normal(gen, (T, H), torch.bfloat16)
        if case["form"] == "all_reduce":
            s.block, s.x, s.residual = blocks[0], x, _normal(gen, (T, H), torch.bfloat16)
        elif W == 1:
            s.block, s.x = blocks[0], x
        else:
            s.op = "mlp_ranks"
            s.shards = [t.clone() for t in x.view(W, T // W, H).unbind(0)]
            s.gate_up = [b.gate_up_packed for b in blocks]
            s.down = [b.down_w for b in blocks]
        return s
    dtype, n = DTYPES[case["dtype"]], case["numel"]
    s.x = s.empty(n, dtype)
    for r in range(case["world"]):
        _fill(gen, w.local(s.x, r))
    s.out = s.empty(n, dtype) if case["out"] == "symmetric" else None
    return s


def _plain(y):
    """Emulated worlds hand back one tensor per rank."""
    return y if isinstance(y, torch.Tensor) else list(y)


_RUN = {
    "all_reduce": lambda s: _plain(tccl.all_reduce(s.x, out=s.out, world=s.world)),
    "all_gather": lambda s: _plain(tccl.all_gather(s.x, world=s.world)),
    "reduce_scatter": lambda s: _plain(tccl.reduce_scatter(s.x, world=s.world)),
    "tree": lambda s: _plain(tccl.double_tree_all_reduce(s.x, world=s.world)),
    "quantized": lambda s: _plain(tccl.quantized_all_reduce(s.x, world=s.world)),
    "gemm": lambda s: gemm_bf16(s.a, s.bt),
    "mlp_sequence": lambda s: s.block.forward(s.x),
    "mlp_all_reduce": lambda s: s.block.forward_allreduce(s.x, residual=s.residual),
    "mlp_ranks": lambda s: tccl.gemm_reduce_scatter(
        tccl.all_gather_gemm(s.shards, s.gate_up, swiglu=True, world=s.world)[0], s.down, world=s.world),
}


def run(state):
    return _RUN[state.op](state)


def work(case):
    op = case["op"]
    if op == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    W = case["world"]
    if op == "mlp":
        T, H, F = case["tokens"], case["hidden"], case["inter"]
        rows = T * H * (3 if case["form"] == "all_reduce" else 2)  # input, output (and the residual)
        return {"bytes": 2 * (rows + 3 * H * F), "flops": 6 * T * H * F}
    size = case["numel"] * SIZE[case["dtype"]]
    moved = {"all_reduce": 2 * W, "tree": 2 * W, "quantized": 2 * W, "reduce_scatter": W + 1, "all_gather": W + W * W}[op]
    adds = {"all_gather": 0, "reduce_scatter": W - 1}.get(op, W - 1)
    return {"bytes": moved * size, "flops": adds * case["numel"]}


def tolerance(case):
    op = case["op"]
    if op in ("gemm", "mlp"):
        return {"rel": 1e-2}  # bf16 operands and results, fp32 sums
    if op == "quantized":
        return {"rel": 2e-2}  # two roundings to e4m3: values at a tie may go the other way
    if op == "all_gather" or case["world"] == 1:
        return "exact"  # copies
    # fp32 sums of `world` terms in any order, one rounding to the data type
    return {"rel": {"bf16": 4e-3, "fp16": 5e-4, "fp32": 1e-6}[case["dtype"]]}
