"""Fused compute + collective ops for tensor parallelism (the "extensible
collectives" the reference names as its motivation — ``presentation.pdf``, slide 4
— but does not implement): GEMM -> reduce-scatter, all-gather -> GEMM, and all-reduce + bias +
residual + RMSNorm.  Each is ONE kernel in which the tensor-core tiles
(tcgen05 / TMEM, fed by TMA from local memory) and the peer traffic (P2P or
NVLS stores / loads over NVLink) overlap tile by tile.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from ..parallel.world import WorldBase
from ..utils import lib as L
from ._common import K, check_sym_tensor, dtype_code, get_world
from .collectives import _planned

__all__ = ["gemm_reduce_scatter", "all_gather_gemm", "all_reduce_bias_residual_rmsnorm", "pack_gate_up",
           "ag_pair_schedule"]


def _locals(w: WorldBase, x):
    """Per-rank local tensors of an ordinary (non symmetric) argument: a tensor in
    a real world, a list/EmuTensor of W tensors in an emulated one."""
    if w.emulated:
        return [x[r] for r in w.local_ranks]
    return [x]  # a real world drives exactly one rank


def _layouts(ts) -> tuple:
    """What a fused kernel's plan depends on in its ordinary operands: everything but the address, of which only the
    alignment matters."""
    return tuple([(t.shape, t.stride(), t.dtype, t.data_ptr() & 15) for t in ts])


def _trace_ptr(w: WorldBase, trace, r: int, grid: int) -> int:
    """``trace``: an int64 CUDA tensor of at least ``grid * 64`` words (a list of them when
    emulated) that receives per-tile %globaltimer stamps; None = no tracing."""
    if trace is None:
        return 0
    t = trace[r] if w.emulated else trace
    if t.dtype != torch.int64 or t.numel() < grid * 64 or not t.is_cuda:
        raise ValueError(f"trace must be an int64 CUDA tensor of >= {grid * 64} words")
    return t.data_ptr()


class FusedPlan:
    """A validated launch of a fused kernel for one layout of its operands: argument structs, one per local rank in
    one array, and the launcher.  Every call writes the addresses of its own operands into the structs, so tensors
    at new addresses cost what known ones do: 11 us of host time for the RMSNorm operator.  (Keyed on addresses it
    was 9 on known ones and 30 on new ones, more than the 18 without any plan.)  ``fresh`` = (shape, strides) of the
    output that a call allocates when the caller gives none; ``views``: buffers of the communicator's own that a call
    hands out.  The structs are shared by all calls of the plan: they are written and launched under one hold of the
    communicator's lock."""

    __slots__ = ("arr", "l", "call", "name", "fresh", "user", "views")

    def __init__(self, w: WorldBase, name: str, arr, grid: int, block: int, extra=(), fresh=None, user=None):
        self.arr, self.name, self.fresh, self.user, self.views = arr, name, fresh, user, None
        self.l = l = L.Launch(grid, block, len(arr) if w.emulated else 0, 0, None)
        fn, refs = getattr(L.lib(), name), (w.comm_ref(), C.byref(arr), *extra, C.byref(l))
        self.call = lambda: fn(*refs)

    def outputs(self, like):
        """New outputs next to the tensors ``like``."""
        shape, strides = self.fresh
        return [torch.empty_strided(shape, strides, dtype=torch.bfloat16, device=t.device) for t in like]

    def go(self, w: WorldBase, device) -> None:
        self.l.stream = torch._C._cuda_getCurrentRawStream(device.index)
        rc = self.call()
        if rc:
            L.check(rc, self.name)
        w.launches += 1


def _gemm_ctas(w: WorldBase, pairs: bool = False) -> int:
    n = w.config.max_ctas or w.num_sms()
    if w.emulated:  # the ranks share one GPU and each CTA takes a whole SM
        n = max(1, w.num_sms() // w.world_size)
    return max(2, n & ~1) if pairs else n


def _stage_handoff(w: WorldBase, user: str) -> bool:
    """Whether a kernel that runs without an entry barrier must take one this time: the staging
    area was last used by a different kernel (every rank sees the same sequence of calls)."""
    last = w.__dict__.get("_stage_user")
    w.__dict__["_stage_user"] = user
    return last != user


def gemm_reduce_scatter(a, bt, out=None, *, trace=None, variant: str = "auto", world: Optional[WorldBase] = None):
    """``out_r = rows r of sum_ranks (a_rank @ bt_rank.T)`` — tensor-parallel
    down-projection fused with the reduce-scatter over token rows.

    ``a``: this rank's ``[M, K_r]`` activations (its slice of the contraction
    dimension), ``bt``: its ``[N, K_r]`` weight slice (``nn.Linear`` layout), both
    bf16.  Returns this rank's ``[M / W, N]`` rows.  ``M % (128 W) == 0`` and
    ``N % 256 == 0``.  Inputs and output are ordinary tensors; the partial tiles
    travel through the communicator's symmetric staging area.

    ``variant``: ``"pair"`` = 256 x 256 tiles on pairs of SMs, the reduction overlapped with the
    mainloop, no entry barrier (needs ``M % (256 W) == 0`` and twice the staging space);
    ``"single"`` = 128 x 256 single-CTA tiles; ``"auto"`` = pair when the shape allows."""
    w = get_world(world)
    As, Bs = _locals(w, a), _locals(w, bt)
    Os = _locals(w, out) if out is not None else None
    key = ("gemm_rs", _layouts(As), _layouts(Bs), Os and _layouts(Os), variant)
    p = _planned(w, key, _plan_gemm_rs, As, Bs, Os, variant)
    grid = p.l.grid
    outs = Os if Os is not None else p.outputs(As)
    with w.lock:
        for g, r, x, b, o in zip(p.arr, w.local_ranks, As, Bs, outs):
            g.a, g.bt, g.out = x.data_ptr(), b.data_ptr(), o.data_ptr()
            g.trace = _trace_ptr(w, trace, r, grid)
        handoff = _stage_handoff(w, p.user)
        p.l.meta = K["TCCL_RS_SYNC_ENTRY"] if handoff and p.user == "gemm_rs_pair" else 0
        p.go(w, As[0].device)
    if out is not None:
        return out
    return outs if w.emulated else outs[0]


def _plan_gemm_rs(w, As, Bs, Os, variant) -> FusedPlan:
    W = w.world_size
    a0, b0 = As[0], Bs[0]
    if a0.dtype != torch.bfloat16 or b0.dtype != torch.bfloat16:
        raise TypeError("gemm_reduce_scatter takes bfloat16 operands")
    M, Kr = a0.shape
    N = b0.shape[0]
    if b0.shape[1] != Kr:
        raise ValueError("a is [M, K], bt is [N, K]")
    if M % (W * 128) or N % 256 or Kr % 8:
        raise ValueError(f"need M % {W * 128} == 0, N % 256 == 0, K % 8 == 0 (got M={M}, N={N}, K={Kr})")
    lib = L.lib()
    for f in ("tccl_gemm_rs_stage_bytes", "tccl_gemm_rs_pair_stage_bytes"):
        getattr(lib, f).restype = C.c_uint64
    stage_bytes = (w.config.stage_mb << 20) - w.ll_bytes
    if variant not in ("auto", "pair", "single"):
        raise ValueError("variant must be 'auto', 'pair' or 'single'")
    pair_ok = M % (W * 256) == 0 and lib.tccl_gemm_rs_pair_stage_bytes(M, N, W) <= stage_bytes
    local = W == 1 and variant != "single"  # one rank: the plain product, no staging area, any row count
    if variant == "pair" and not pair_ok:
        raise ValueError(f"the pair kernel needs M % {W * 256} == 0 and "
                         f"{lib.tccl_gemm_rs_pair_stage_bytes(M, N, W) >> 20} MiB of staging area")
    pair = (pair_ok or local) and variant != "single"
    need = 0 if local else lib.tccl_gemm_rs_pair_stage_bytes(M, N, W) if pair else lib.tccl_gemm_rs_stage_bytes(M, N, W)
    if need > stage_bytes:
        raise ValueError(f"staging area too small: need {need >> 20} MiB, have {w.config.stage_mb} MiB "
                         "(raise TCCL_STAGE_MB)")
    arr = (L.GemmRsArgs * len(As))()
    for i, (ar, br) in enumerate(zip(As, Bs)):
        if ar.stride(1) != 1 or br.stride(1) != 1:
            raise ValueError("operands must have a unit inner stride")
        ldo = Os[i].stride(0) if Os is not None else N
        arr[i] = L.GemmRsArgs(0, 0, 0, M, N, Kr, ar.stride(0), br.stride(0), ldo, 0)
    name = "tccl_gemm_reduce_scatter_pair" if pair else "tccl_gemm_reduce_scatter"
    return FusedPlan(w, name, arr, _gemm_ctas(w, pair), 256, (C.c_uint64(stage_bytes),), ((M // W, N), (N, 1)),
                     "gemm_rs_pair" if pair else "gemm_rs")


def ag_pair_schedule(W: int, rank: int, tm: int, tn: int, pairs: int, nbatch: int, k: int, *, halves: bool = True,
                     ring: bool = False, pair_tflops: float = 20.0, link_gbs: float = 600.0, start_us: float = 8.0,
                     round_us: float = 2.0):
    """Plan of the all-gather -> GEMM pair kernel: for every CTA pair the tiles it runs, in order.

    The kernel's built-in order deals tile ``pair + i * pairs`` to a pair whatever the moment its rows
    arrive; at 8 ranks most pairs then sit on a remote tile while others queue two tiles behind theirs.
    This is list scheduling against a small cost model instead: the rank's own rows are there at once,
    batch ``b`` of the peers' rows (``nbatch`` batches of ``tm / nbatch`` 128-row tiles per rank) after
    ``start_us + (b + 1) / nbatch`` of the time the link needs for all of them (``ring``: the movers send
    destination by destination, so the rows of rank ``rank - j`` are there after ``j`` rounds of one shard
    each plus ``round_us`` per round), a 256 x 256 tile costs ``2 * 256 * 256 * k / pair_tflops``.  Tiles are taken in the order their rows arrive and handed to
    the pair that is free first; the last tiles (those of the last batch, one wave at most) are cut into
    256 x 128 halves so that the work left when the last rows land spreads over all pairs.  Returns
    ``pairs`` lists of ``(mt, nt, half)`` (``mt`` = even 128-row tile index, ``half`` 0 / 1 / 2 = whole
    tile / left / right half).  Any plan that names every tile once is correct — the kernel waits for
    the rows of whatever tile it is given — the model only decides how good it is."""
    import heapq

    tm2 = tm // 2
    rows_in = (W - 1) * tm * 128
    link_us = rows_in * k * 2 / (link_gbs * 1e3)
    arrive = [start_us + (b + 1) / nbatch * link_us for b in range(nbatch)]
    tile_us = 2.0 * 256 * 256 * k / (pair_tflops * 1e6)
    units = []  # (ready, mt, nt, group): group = batch (or round) the rows come with, -1 = own
    for rt2 in range(tm2):
        for nt in range(tn):
            units.append((0.0, rank * tm + 2 * rt2, nt, -1))
    last = nbatch - 1
    if ring:
        shard_us = tm * 128 * k * 2 / (link_gbs * 1e3)
        last = W - 1
        for j in range(1, W):
            src = (rank - j) % W
            for rt2 in range(tm2):
                for nt in range(tn):
                    units.append((start_us + j * (shard_us + round_us), src * tm + 2 * rt2, nt, j))
    else:
        for rt2 in range(tm2):
            b = min(nbatch - 1, (2 * rt2 + 1) * nbatch // tm)
            for j in range(1, W):
                src = (rank + j) % W
                for nt in range(tn):
                    units.append((arrive[b], src * tm + 2 * rt2, nt, b))
    units.sort(key=lambda u: u[0])  # stable: own rows, then batch by batch
    n_last = sum(1 for u in units if u[3] == last)
    split_from = len(units) - min(n_last, pairs) if (halves and W > 1) else len(units)
    free = [(0.0, p) for p in range(pairs)]
    heapq.heapify(free)
    plan = [[] for _ in range(pairs)]
    for idx, (ready, mt, nt, _) in enumerate(units):
        parts = ((0, tile_us),) if idx < split_from else ((1, tile_us / 2 + 1.0), (2, tile_us / 2 + 1.0))
        for half, dur in parts:
            t, p = heapq.heappop(free)
            plan[p].append((mt, nt, half))
            heapq.heappush(free, (max(t, ready) + dur, p))
    return plan


def _ag_sched_tensor(w, r: int, tm: int, tn: int, pairs: int, nbatch: int, k: int, halves: bool, device):
    cache = w.__dict__.setdefault("_ag_sched", {})
    cfg = w.config
    key = (r, tm, tn, pairs, nbatch, k, halves, bool(cfg.ag_ring), cfg.ag_pair_tflops, cfg.ag_link_gbs)
    t = cache.get(key)
    if t is None:
        plan = ag_pair_schedule(w.world_size, r, tm, tn, pairs, nbatch, k, halves=halves, ring=bool(cfg.ag_ring),
                                pair_tflops=cfg.ag_pair_tflops, link_gbs=cfg.ag_link_gbs)
        stride = max(len(x) for x in plan) + 1
        rows = [[m | (n << 12) | (h << 28) for (m, n, h) in x] + [-1] * (stride - len(x)) for x in plan]
        t = cache[key] = torch.tensor(rows, dtype=torch.int32).to(device)
    return t


def all_gather_gemm(a_shard, bt, a_full=None, out=None, *, comm_ctas: int = 0, swiglu: bool = False, trace=None,
                    lsu_movers: bool = False, variant: str = "auto", world: Optional[WorldBase] = None):
    """``out_r = all_gather(a_shard) @ bt_r.T`` — tensor-parallel up-projection
    fused with the all-gather of the token rows.

    ``a_shard``: this rank's ``[M / W, K]`` rows (bf16, any device memory), ``bt``:
    its ``[N_r, K]`` weight slice.  ``a_full`` is the ``[M, K]`` gathered buffer in
    symmetric memory (allocated and cached per shape when omitted); it holds the
    gathered activations afterwards.  Returns ``(out, a_full)`` with ``out`` the
    rank's ``[M, N_r]`` result.  ``M % (128 W) == 0``.

    ``swiglu=True`` fuses the gated activation into the epilogue: ``bt`` must be
    packed by :func:`pack_gate_up` (every 256-row block = 128 gate rows, then the
    128 matching up rows) and ``out`` is ``[M, N_r / 2] = silu(gate) * up``.

    ``variant``: ``"pair"`` = 256 x 256 tiles on pairs of SMs, every CTA moves its share of the
    shard before it computes (needs ``M % (256 W) == 0``); ``"single"`` = 128 x 256 single-CTA
    tiles with ``comm_ctas`` dedicated data movers; ``"auto"`` = pair when the shape allows.  When
    the pair kernel allocates the gathered buffer itself it keeps two of them and alternates (so it
    needs no barrier on entry): the returned ``a_full`` is the one this call filled, and it stays
    valid until the call after the next one."""
    w = get_world(world)
    As, Bs = _locals(w, a_shard), _locals(w, bt)
    Os = _locals(w, out) if out is not None else None
    opts = (a_full is None, comm_ctas, swiglu, int(lsu_movers), variant)
    key = ("ag_gemm", _layouts(As), _layouts(Bs), Os and _layouts(Os), opts)
    p = _planned(w, key, _plan_ag_gemm, As, Bs, Os, *opts)
    grid = p.l.grid
    outs = Os if Os is not None else p.outputs(As)
    full_ptrs, mc, seq = None, 0, 0
    if a_full is not None:
        full_ptrs, mc = w.peer_ptrs(a_full), _ag_multicast(w, a_full, p.user == "ag_gemm_pair")
    with w.lock:
        for g, r, x, b, o in zip(p.arr, w.local_ranks, As, Bs, outs):
            g.a_shard, g.bt, g.out = x.data_ptr(), b.data_ptr(), o.data_ptr()
            g.trace = _trace_ptr(w, trace, r, grid)
            if full_ptrs is not None:
                g.a_full[: len(full_ptrs)] = full_ptrs
                g.mc_a_full = mc
        p.go(w, As[0].device)
        if p.user == "ag_gemm_pair":  # mirrors the device's count of pair calls, which picks the half (see reset())
            seq = w.__dict__.get("_ag_seq", 0)
            w.__dict__["_ag_seq"] = seq + 1
    res = out if out is not None else (outs if w.emulated else outs[0])
    return res, (a_full if a_full is not None else p.views[seq % len(p.views)])


def _ag_multicast(w, a_full, pair) -> int:
    # two ranks: the switch would deliver every row to its sender too (twice the inbound bytes of a plain store)
    return w.mc_ptr(a_full) if ((w.world_size > 2 and not w.config.ag_ring) or not pair) else 0


def _plan_ag_gemm(w, As, Bs, Os, own_full, comm_ctas, swiglu, lsu_movers, variant) -> FusedPlan:
    W = w.world_size
    a0, b0 = As[0], Bs[0]
    if a0.dtype != torch.bfloat16 or b0.dtype != torch.bfloat16:
        raise TypeError("all_gather_gemm takes bfloat16 operands")
    rows, Kd = a0.shape
    M, N = rows * W, b0.shape[0]
    if b0.shape[1] != Kd:
        raise ValueError("a_shard is [M / W, K], bt is [N, K]")
    if rows % 128 or N % 8 or Kd % 8:
        raise ValueError(f"need (M / W) % 128 == 0, N % 8 == 0, K % 8 == 0 (got M/W={rows}, N={N}, K={Kd})")
    if swiglu and N % 256:
        raise ValueError("swiglu needs N % 256 == 0 (whole gate|up tiles)")
    n_out = N // 2 if swiglu else N
    if variant not in ("auto", "pair", "single"):
        raise ValueError("variant must be 'auto', 'pair' or 'single'")
    pair_ok = rows % 256 == 0
    if variant == "pair" and not pair_ok:
        raise ValueError("the pair kernel needs (M / W) % 256 == 0")
    # one rank: the last pair tile may hang over the end of the rows
    pair = (pair_ok or (W == 1 and variant == "auto")) and variant != "single"
    half_bytes = 0
    views, full_ptrs, mc = None, (), 0
    if own_full:
        cache = w.__dict__.setdefault("_ag_buffers", {})
        key = (M, Kd, pair)
        a_full = cache.get(key)
        if a_full is None:
            a_full = cache[key] = w.empty((2, M, Kd) if pair else (M, Kd), torch.bfloat16)
        half = a_full.half if w.emulated else a_full.__getitem__
        views = [half(0), half(1)] if pair else [a_full]
        half_bytes = M * Kd * 2 if pair else 0
        full_ptrs, mc = w.peer_ptrs(a_full), _ag_multicast(w, a_full, pair)
    grid = _gemm_ctas(w, pair)
    if comm_ctas <= 0:
        # Few data movers: every mover CTA is an SM the GEMM does not get, and 8 movers
        # with 8 vectors per thread in flight already fill the link (measured on 8xB200,
        # Llama-3-8B up-projection: 8 movers 116 us, 16: 121 us, 24: 125 us, 48: 128 us).
        comm_ctas = w.config.ag_movers if grid > 16 else 2
        comm_ctas = max(1, min(comm_ctas, grid - 1))
    arr = (L.AgGemmArgs * len(As))()
    for i, (r, ar, br) in enumerate(zip(w.local_ranks, As, Bs)):
        if ar.stride(1) != 1 or br.stride(1) != 1:
            raise ValueError("operands must have a unit inner stride")
        ldo = n_out
        if Os is not None:
            o = Os[i]
            if o.shape != (M, n_out) or o.dtype != torch.bfloat16 or o.stride(1) != 1:
                raise ValueError(f"out must be bf16 [{M}, {n_out}] with a unit inner stride")
            ldo = o.stride(0)
        g = arr[i]
        for q, v in enumerate(full_ptrs):
            g.a_full[q] = v
        g.mc_a_full = mc
        g.m, g.n, g.k = M, N, Kd
        g.lda_shard, g.lda_full, g.ldb, g.ldo = ar.stride(0), Kd, br.stride(0), ldo
        g.comm_ctas = max(1, int(w.config.ag_batches)) if pair else comm_ctas  # pair kernel: batches of the mover phase
        g.swiglu = 1 if swiglu else 0
        g.lsu_movers = lsu_movers
        if pair:  # bits: 2 = move the shard only (timeline tool), 4 = movers send destination by destination
            g.lsu_movers = (2 if lsu_movers == 2 else 0) | (4 if w.config.ag_ring else 0)
        if pair and w.config.ag_schedule and W > 1:
            nb = max(1, min(int(w.config.ag_batches), rows // 128))
            sched = _ag_sched_tensor(w, r, rows // 128, -(-N // 256), grid // 2, nb, Kd, True, ar.device)
            g.sched, g.sched_stride = sched.data_ptr(), sched.shape[1]
    p = FusedPlan(w, "tccl_allgather_gemm_pair" if pair else "tccl_allgather_gemm", arr, grid, 256,
                  (C.c_uint64(half_bytes),) if pair else (), ((M, n_out), (n_out, 1)), "ag_gemm_pair" if pair else "ag_gemm")
    p.views = views
    return p


def all_reduce_bias_residual_rmsnorm(x, weight, bias=None, residual=None, eps: float = 1e-5, out=None,
                                     residual_out=None, *, algo: str = "auto", world: Optional[WorldBase] = None):
    """``y = RMSNorm(all_reduce(x) + bias + residual) * weight`` in one kernel.

    ``x``: this rank's partial ``[tokens, hidden]`` in symmetric memory (the output
    of a row-parallel linear before its reduction).  ``bias`` / ``weight``:
    ``[hidden]``; ``residual``: this rank's (replicated) ``[tokens, hidden]``.
    ``out`` (and ``residual_out``, the pre-norm sum that becomes the next residual)
    live in symmetric memory because every rank writes its rows into all of them;
    they are allocated and cached per shape when omitted (pass ``residual_out=True``
    to ask for the pre-norm sum).  Returns ``y`` or ``(y, residual_out)``."""
    w = get_world(world)
    want_res = residual_out is not None and residual_out is not False
    given = residual_out if want_res and residual_out is not True else None
    Ws, Bs, Rs = _locals(w, weight), (_locals(w, bias) if bias is not None else None), \
        (_locals(w, residual) if residual is not None else None)
    # the caller's symmetric tensors: checked, and their addresses taken, on every call
    xp, op, rp = [None if t is None else check_sym_tensor(w, t, what)
                  for t, what in ((x, "input"), (out, "out"), (given, "residual_out"))]
    x0, eps = w.local(x, w.local_ranks[0]), float(eps)
    key = ("arn", x0.shape, x0.dtype, _layouts(Ws), Bs and _layouts(Bs), Rs and _layouts(Rs), eps, out is None, want_res,
           given is None, algo)
    p = _planned(w, key, _plan_arn, x0, Ws, Bs, Rs, eps, out is None, want_res, given is None, algo)
    W = w.world_size
    with w.lock:
        for i, a in enumerate(p.arr):
            a.x[:W], a.mc_x = xp, w.mc_ptr(x)
            if op is not None:
                a.out[:W], a.mc_out = op, w.mc_ptr(out)
            if rp is not None:
                a.res_out[:W], a.mc_res_out = rp, w.mc_ptr(given)
            a.weight = Ws[i].data_ptr()
            if Bs is not None:
                a.bias = Bs[i].data_ptr()
            if Rs is not None:
                a.residual = Rs[i].data_ptr()
        p.go(w, Ws[0].device)
    if out is None:
        out = p.views[0]
    return (out, p.views[1] if given is None else given) if want_res else out


def _plan_arn(w, x0, Ws, Bs, Rs, eps, own_out, want_res, own_res, algo) -> FusedPlan:
    if x0.dim() != 2:
        raise ValueError("x must be [tokens, hidden]")
    T, H = x0.shape
    dt = dtype_code(x0.dtype)
    vpt = 16 // x0.element_size()
    if H % vpt or H > 512 * 4 * vpt:
        raise ValueError(f"hidden must be a multiple of {vpt} and at most {512 * 4 * vpt}")
    cache = w.__dict__.setdefault("_arn_buffers", {})

    def sym(tag):
        key = (tag, T, H, x0.dtype)
        if key not in cache:
            cache[key] = w.empty((T, H), x0.dtype)
        return cache[key]

    out = sym("out") if own_out else None
    res_out = sym("residual_out") if want_res and own_res else None
    if algo == "auto":
        algo = "nvls" if w.has_nvls and w.world_size > 2 else "p2p"
    if algo == "nvls" and not w.has_nvls:
        raise RuntimeError("nvls variant needs NVLS multicast")
    arr = (L.ArnArgs * len(w.local_ranks))()
    for i, a in enumerate(arr):
        if out is not None:
            a.out[: w.world_size], a.mc_out = w.peer_ptrs(out), w.mc_ptr(out)
        if res_out is not None:
            a.res_out[: w.world_size], a.mc_res_out = w.peer_ptrs(res_out), w.mc_ptr(res_out)
        for name, src in (("weight", Ws), ("bias", Bs), ("residual", Rs)):
            if src is None:
                continue
            tns = src[i]
            if tns.dtype != x0.dtype or not tns.is_contiguous() or tns.data_ptr() % 16:
                raise ValueError(f"{name} must be contiguous, 16-byte aligned and of x's dtype")
            if tns.numel() != (T * H if name == "residual" else H):
                raise ValueError(f"{name} has the wrong size")
        a.eps, a.tokens, a.hidden, a.dtype = float(eps), T, H, dt
        a.flags = w.coll_flags()
    rows = -(-T // w.world_size)
    nv = H // vpt
    per_sm = 2 if nv <= 512 and not w.emulated else 1  # narrow rows: two CTAs per SM
    batch = 1                                          # rows a CTA handles together (kernel's R)
    grid = max(1, min(-(-rows // batch), w.max_ctas() * per_sm, K["TCCL_MAX_BLOCKS"]))
    p = FusedPlan(w, "tccl_allreduce_bias_residual_rmsnorm", arr, grid, 512, (1 if algo == "nvls" else 0,))
    p.views = (out, res_out)
    return p


def pack_gate_up(gate_w: torch.Tensor, up_w: torch.Tensor) -> torch.Tensor:
    """Interleave ``gate_w`` and ``up_w`` (both ``[F, K]``, ``F % 128 == 0``) in
    blocks of 128 rows — gate rows ``[128 j, 128 j + 128)`` followed by the same
    rows of ``up_w`` — which is the weight layout the ``swiglu`` epilogue of
    :func:`all_gather_gemm` expects (one 256-wide output tile = 128 gate columns
    and the 128 up columns they multiply)."""
    F, Kd = gate_w.shape
    if up_w.shape != gate_w.shape or F % 128:
        raise ValueError("gate and up weights must both be [F, K] with F % 128 == 0")
    return torch.stack([gate_w.view(F // 128, 128, Kd), up_w.view(F // 128, 128, Kd)], dim=1).reshape(2 * F, Kd).contiguous()
