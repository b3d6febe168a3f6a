"""What the native launchers refuse, in real and in emulated mode.  A launch that is not refused needs a GPU: without one
it comes back with a CUDA error (positive), a refused one with a code of this library (negative)."""
import ctypes as C

import pytest

from tccl_b200.ops.quantized import QarArgs
from tccl_b200.utils import lib as L

K = L.K
GOOD = 0x1000  # an aligned address; nothing is launched


def _comms(W):
    comms = (L.Comm * W)()
    for r, c in enumerate(comms):
        c.world, c.rank = W, r
        c.stage_bytes, c.ll_bytes, c.timeout_ns = 64 << 20, 2 << 20, 1000
        c.tree_bytes = K["TCCL_TREE_LL_BYTES"] + 4 * 8 * K["TCCL_TREE_RING_DEPTH"] * K["TCCL_TREE_SLICE_BYTES"]
    return comms


def _tree(W, **kw):
    a = (L.TreeArgs * W)()
    for x in a:
        x.numel, x.chunk_vecs, x.dtype, x.ctas_per_role = 1 << 16, 64, K["TCCL_F32"], 2
    return a


def _qar(W, **kw):
    return (QarArgs * W)(*[QarArgs(GOOD, GOOD, 2048 * 64, 0) for _ in range(W)])


def _coll(W, **kw):
    a = (L.CollArgs * W)()
    for x in a:
        x.numel, x.dtype, x.flags = 4096, K["TCCL_F32"], kw.get("flags", 0)
        for p in range(W):
            x.inp[p] = x.out_peer[p] = GOOD
    return a


PIPE = (8 << K["TCCL_F_PIPE_REDUCERS_SHIFT"]) | (3 << K["TCCL_F_PIPE_STAGES_SHIFT"]) | (4 << K["TCCL_F_PIPE_UNROLL_SHIFT"])
CASES = {  # launcher -> (args, launch, what makes one rank's struct wrong)
    "tccl_allreduce_tree": (_tree, dict(grid=8, block=512), dict(
        slice_beyond_its_ring_slot=lambda c, a: setattr(a, "chunk_vecs", 2 * K["TCCL_TREE_SLICE_BYTES"] // 16 + 1),
        no_chunk=lambda c, a: setattr(a, "chunk_vecs", 0),
        more_pipelines_than_the_ring=lambda c, a: setattr(c, "tree_bytes", K["TCCL_TREE_LL_BYTES"]),
        grid_of_other_pipelines=lambda c, a: setattr(a, "ctas_per_role", 3))),
    "tccl_allreduce_tree_ll": (_tree, dict(grid=8, block=512), dict(
        more_than_the_slots=lambda c, a: setattr(a, "numel", 1 << 24),
        no_ring=lambda c, a: setattr(c, "tree_bytes", 0),
        ragged=lambda c, a: setattr(a, "numel", 1023))),
    "tccl_allreduce_fp8wire": (_qar, dict(grid=8, block=256), dict(
        ragged=lambda c, a: setattr(a, "numel", 2047),
        off_the_vector_grid=lambda c, a: setattr(a, "out", GOOD + 2),
        staging_area_too_small=lambda c, a: setattr(c, "stage_bytes", 1 << 10))),
    "tccl_allreduce_twoshot_bulk": (_coll, dict(grid=8, block=256), dict(
        off_the_vector_grid=lambda c, a: a.inp.__setitem__(0, GOOD + 8))),
    "tccl_allreduce_twoshot_pipe_p2p": (lambda W: _coll(W, flags=PIPE), dict(grid=8, block=512, meta=PIPE), dict(
        another_pipeline=lambda c, a: setattr(a, "flags", 0))),
}


def _launch(name, comms, args, W, emulated, grid, block, meta=0):
    l = L.Launch(grid, block, W if emulated else 0, meta, None)
    return getattr(L.lib(), name)(C.byref(comms), C.byref(args), C.byref(l))


@pytest.mark.parametrize("name,wrong", [(n, w) for n, (_, _, ws) in CASES.items() for w in ws])
def test_every_rank_is_checked(name, wrong):
    make, launch, wrongs = CASES[name]
    comms, args = _comms(2), make(2)
    wrongs[wrong](comms[0], args[0])
    assert _launch(name, comms, args, 2, False, **launch) < 0
    for r in (0, 1):  # emulated: every rank's struct
        comms, args = _comms(2), make(2)
        wrongs[wrong](comms[r], args[r])
        assert _launch(name, comms, args, 2, True, **launch) < 0, r


@pytest.mark.parametrize("name", sorted(CASES))
def test_emulated_launch_of_another_world_is_refused(name):
    """Ranks that are not launched would be waited for."""
    make, launch, _ = CASES[name]
    assert _launch(name, _comms(4), make(4), 2, True, **launch) < 0
    assert _launch(name, _comms(2), make(2), -1, True, **launch) < 0
    assert _launch(name, _comms(2), make(2), L.MAX_WORLD + 1, True, **launch) < 0


@pytest.mark.parametrize("name", ["tccl_allreduce_oneshot_p2p", "tccl_allreduce_twoshot_p2p", "tccl_reducescatter_p2p",
                                  "tccl_allgather_pull_p2p", "tccl_allreduce_push_p2p", "tccl_allreduce_oneshot_nvls"])
def test_world_sizes_without_a_kernel_are_refused(name):
    for world in (0, -1, L.MAX_WORLD + 1):
        comms, args = _comms(1), _coll(1)
        comms[0].world = world
        assert _launch(name, comms, args, 1, False, grid=8, block=512) < 0
