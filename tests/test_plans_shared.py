"""What cached launches share between calls, on the CPU with a stub in place of the native launchers: host threads that
call one operator on the same operands, and what keeps a communicator alive."""
import ctypes as C
import gc
import sys
import threading
import time
import weakref

import pytest
import torch

from tccl_b200.config import Config
from tccl_b200.ops import collectives, fused, quantized
from tccl_b200.ops import tree_allreduce
from tccl_b200.parallel.emu import EmuTensor, EmuWorld
from tccl_b200.parallel.world import RealWorld
from tccl_b200.utils import lib as L

_here = threading.local()  # .stream: what the calling thread uses as its current stream


class StubLib:
    """The real library, but launchers only note what they were given: (name, outputs, stream).  Like a call through
    ctypes they let other threads run before they look at the structs."""

    def __init__(self, real):
        self._real, self.seen = real, []

    def __getattr__(self, name):
        if "stage_bytes" in name or "chunk_bytes" in name or "max_ctas" in name or "error" in name:
            return getattr(self._real, name)

        def launch(*refs):
            time.sleep(0)
            args, l = refs[1]._obj, refs[-1]._obj
            structs = list(args) if isinstance(args, C.Array) else [args]
            self.structs = [type(s).from_buffer_copy(s) for s in structs]
            self.seen.append((name, [s.out if isinstance(s.out, int) else s.out[r] for r, s in enumerate(structs)], l.stream or 0))
            return 0

        return launch


@pytest.fixture
def stub(monkeypatch):
    s = StubLib(L.lib())
    monkeypatch.setattr(L, "lib", lambda: s)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda dev: getattr(_here, "stream", 7), raising=False)
    for m in (collectives, fused, tree_allreduce):
        monkeypatch.setattr(m, "check_sym_tensor", lambda w, x, *a: w.peer_ptrs(x))
    return s


def one_rank(stub):
    """A one-rank communicator over ordinary CPU memory."""
    class World(RealWorld):
        def __init__(self):
            self._test_setup()

        def _resolve(self, t):
            return [t.data_ptr()], 0

        def empty(self, shape, dtype=torch.bfloat16):
            return torch.empty(shape, dtype=dtype)

        def _test_setup(self):
            self.config = Config()
            self.world_size, self.rank, self._nvls, self._sms = 1, 0, False, 148
            self.device = torch.device("cuda", 0)
            self.ll_bytes, self.comm, self._handles = 2 << 20, L.Comm(), {}
            self._start_plans()

    return World()


def emulated(stub, W):
    w = object.__new__(EmuWorld)
    w.world_size, w.config, w._sms, w.device = W, Config(), 148, torch.device("cuda", 0)
    w._stage_bytes, w.ll_bytes, w.tree_bytes = 64 << 20, 2 << 20, 0
    w.comms = (L.Comm * W)()
    w.empty = lambda shape, dtype=torch.bfloat16: EmuTensor([torch.empty(shape, dtype=dtype) for _ in range(W)])
    w._start_plans()
    return w


def _two_threads(fn, calls=400):
    """Outputs returned to two threads that call ``fn`` at the same time, each on a stream of its own."""
    got, errors = [[], []], []
    gate = threading.Barrier(2)

    def body(k):
        _here.stream = 100 + k
        try:
            gate.wait()
            for _ in range(calls):
                got[k].append(fn())
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    old = sys.getswitchinterval()
    sys.setswitchinterval(1e-5)
    try:
        ts = [threading.Thread(target=body, args=(k,)) for k in (0, 1)]
        [t.start() for t in ts]
        [t.join() for t in ts]
    finally:
        sys.setswitchinterval(old)
    assert not errors, errors[0]
    return got


def _ptrs(y):
    return [t.data_ptr() for t in (y if isinstance(y, (list, EmuTensor)) else [y])]


def _bf16(*shape):
    return torch.zeros(shape, dtype=torch.bfloat16)


CALLS = {
    "gemm_reduce_scatter": lambda w, ops: fused.gemm_reduce_scatter(ops["a"], ops["b"], world=w),
    "all_gather_gemm": lambda w, ops: fused.all_gather_gemm(ops["a"], ops["b"], world=w)[0],
    "quantized_all_reduce": lambda w, ops: quantized.quantized_all_reduce(ops["x"], world=w),
    "all_reduce_bias_residual_rmsnorm": lambda w, ops: fused.all_reduce_bias_residual_rmsnorm(ops["n"], ops["g"], world=w),
    "all_reduce": lambda w, ops: collectives.all_reduce(ops["x"], world=w),
    "all_gather": lambda w, ops: collectives.all_gather(ops["x"], world=w),
}


def _operands(w):
    W = w.world_size
    shapes = {"a": (256 * W, 64), "b": (256, 64), "x": (4096,), "n": (4, 1024), "g": (1024,)}
    if not w.emulated:
        return {k: _bf16(*s) for k, s in shapes.items()}
    return {k: EmuTensor([_bf16(*s) for _ in range(W)]) for k, s in shapes.items()}


@pytest.mark.parametrize("world", ["one rank", "emulated"])
@pytest.mark.parametrize("op", sorted(CALLS))
def test_two_threads_never_share_a_launch(stub, op, world):
    """Every output that a call hands out was given to a launch of its own, on the calling thread's stream."""
    w = one_rank(stub) if world == "one rank" else emulated(stub, 2)
    ops = _operands(w)
    got = _two_threads(lambda: CALLS[op](w, ops))
    seen = {(tuple(outs), stream) for _, outs, stream in stub.seen}
    missing = [(k, y) for k in (0, 1) for y in got[k] if (tuple(_ptrs(y)), 100 + k) not in seen]
    assert not missing, f"{len(missing)} of {len(got[0]) + len(got[1])} outputs were in no launch of their thread"
    streams = [stream for _, _, stream in stub.seen]
    assert [streams.count(100), streams.count(101)] == [len(got[0]), len(got[1])] and w.launches == len(streams)


@pytest.mark.parametrize("world", ["one rank", "emulated"])
def test_a_dropped_communicator_is_freed_at_once(stub, world):
    """Cached launches do not keep their communicator (and its device memory) alive: no cycle for the collector to find."""
    w = one_rank(stub) if world == "one rank" else emulated(stub, 2)
    ops = _operands(w)
    for _ in range(2):
        for op in sorted(CALLS):
            CALLS[op](w, ops)
    x = ops["x"]
    collectives.all_reduce(x, inplace=True, algo="oneshot_p2p", world=w)
    w.config.oneshot_max_bytes = 16
    w.config.push_max_bytes = 16
    collectives.all_reduce(x, world=w)                                        # staged: a symmetric buffer, then a copy
    collectives.all_reduce(x, out=_like(w, x), algo="oneshot_p2p", world=w)
    gone, had_gc = weakref.ref(w), gc.isenabled()
    gc.disable()
    try:
        del w
        assert gone() is None
    finally:
        if had_gc:
            gc.enable()


def _like(w, x):
    return EmuTensor([p.clone() for p in x.parts]) if w.emulated else x.clone()


@pytest.mark.parametrize("world", ["one rank", "emulated"])
def test_fused_operators_plan_once_per_layout(stub, world):
    """Operands at new addresses reach the launcher without a new plan; a layout that is refused stays refused after a
    good one of the same shape was planned."""
    w = one_rank(stub) if world == "one rank" else emulated(stub, 2)
    W, ranks = w.world_size, w.local_ranks
    fields = {"gemm_reduce_scatter": {"a": "a", "bt": "b"}, "all_gather_gemm": {"a_shard": "a", "bt": "b"},
              "quantized_all_reduce": {"inp": "x"}, "all_reduce_bias_residual_rmsnorm": {"weight": "g", "x": "n"}}
    keep = []  # new addresses, not reused ones
    for op, names in fields.items():
        sizes = set()
        for _ in range(3):
            ops = _operands(w)
            keep.append(ops)
            CALLS[op](w, ops)
            sizes.add(len(w.plans))
            for r, s in zip(ranks, stub.structs):
                for f, k in names.items():
                    got, want = getattr(s, f), [w.local(ops[k], q).data_ptr() for q in ranks]
                    assert (got == want[r]) if isinstance(got, int) else (list(got)[:W] == want), (op, f)
        assert len(sizes) == 1, f"{op}: {sizes} plans"
    emu = lambda f: EmuTensor([f() for _ in range(W)]) if w.emulated else f()  # noqa: E731
    off = lambda *shape: _bf16(8 + int(torch.tensor(shape).prod()))[1: 1 + int(torch.tensor(shape).prod())].view(shape)  # noqa: E731
    with pytest.raises(ValueError):  # 2 bytes off the 16-byte grid
        CALLS["quantized_all_reduce"](w, {"x": emu(lambda: off(4096))})
    with pytest.raises(ValueError):
        CALLS["quantized_all_reduce"](w, {"x": emu(lambda: _bf16(2, 8192)[:, :2048])})
    with pytest.raises(ValueError):
        CALLS["all_reduce_bias_residual_rmsnorm"](w, {"n": keep[0]["n"], "g": emu(lambda: off(1024))})
    with pytest.raises(ValueError):
        CALLS["gemm_reduce_scatter"](w, {"a": emu(lambda: _bf16(64, 256 * W).t()), "b": keep[0]["b"]})
    with pytest.raises(TypeError):
        CALLS["all_gather_gemm"](w, {"a": emu(lambda: torch.zeros(256 * W, 64, dtype=torch.float16)), "b": keep[0]["b"]})


def test_fused_operators_write_the_callers_buffers(stub):
    """Symmetric tensors that the caller passes reach the launcher at their addresses of this call."""
    w = one_rank(stub)
    for _ in range(2):
        ops, y, res, full = _operands(w), _bf16(4, 1024), _bf16(4, 1024), _bf16(256, 64)
        assert fused.all_reduce_bias_residual_rmsnorm(ops["n"], ops["g"], residual=ops["n"], out=y, residual_out=res, world=w) == (y, res)
        s, = stub.structs
        assert (s.out[0], s.res_out[0], s.residual, s.bias) == (y.data_ptr(), res.data_ptr(), ops["n"].data_ptr(), 0)
        out, got = fused.all_gather_gemm(ops["a"], ops["b"], a_full=full, world=w)
        s, = stub.structs
        assert got is full and s.a_full[0] == full.data_ptr() and s.out == out.data_ptr()
        fused.all_reduce_bias_residual_rmsnorm(ops["n"], ops["g"], world=w)
        s, = stub.structs
        assert s.residual == 0 and s.res_out[0] == 0


def test_plan_cache_lookups_race_with_evictions():
    """Lookups take no lock: a plan that goes away in the middle of one is no error."""
    from tccl_b200.parallel.world import PlanCache

    class Evicting(PlanCache):
        def get(self, key):  # another thread evicts the plan between the two steps of a lookup
            p = super().get(key)
            self.pop(key, None)
            return p

    cache = Evicting(4)
    cache.insert("a", 1)
    assert cache.lookup("a") == 1 and cache.lookup("a") is None


@pytest.mark.parametrize("wrong", ["dtype", "stride"])
def test_a_destination_of_another_layout_is_refused_on_every_rank(stub, wrong):
    """A cached launch must not swallow the check of any rank's destination: here rank 1's, at the same address as a good
    one that was planned before."""
    w = emulated(stub, 2)
    x, shares = EmuTensor([_bf16(4096) for _ in range(2)]), [_bf16(4096) for _ in range(2)]
    bad = shares[1].view(torch.float16) if wrong == "dtype" else shares[1].as_strided((2048,), (2,))
    cases = [(lambda out: collectives.all_reduce(x, out=out, algo="oneshot_p2p", world=w), 4096),
             (lambda out: collectives.reduce_scatter(x, out=out, world=w), 2048)]
    for call, n in cases:
        call(EmuTensor([s[:n] for s in shares]))
        with pytest.raises(ValueError):
            call(EmuTensor([shares[0][:n], bad[:n]]))
    half = [_bf16(2048) for _ in range(2)]
    collectives.all_gather(EmuTensor(half), out=EmuTensor(shares), algo="pull", world=w)
    with pytest.raises(ValueError):
        collectives.all_gather(EmuTensor(half), out=EmuTensor([shares[0], bad]), algo="pull", world=w)
