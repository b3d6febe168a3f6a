"""The kernel for few rows (``gemm_skinny.cu``) in every configuration there is, whichever one the cost model would pick."""
import ctypes as C
import itertools
import random

import pytest
import torch

from tccl_b200.utils import lib as L

# (tokens, CTAs) of a tile; K split 1 .. 8 ways over a cluster of at most 8 CTAs; two CTAs on an SM up to 128 tokens
TILES = [(16, 1), (32, 1), (64, 1), (128, 1), (32, 2), (64, 2), (128, 2), (256, 2)]
CONFIGS = [(tn, cg, s, per) for tn, cg in TILES for s in (1, 2, 4, 8) if cg * s <= 8 for per in (1, 2) if tn <= 128 or per == 1]


def choice(m, n, k):
    f = L.FewRows()
    assert L.lib().tccl_gemm_choice(m, n, k, C.byref(f)) == 0
    return f.tokens, f.ctas, f.splits, f.per_sm


def test_choices_are_among_the_configurations_that_are_tested():
    """Over the range of shapes that the operator takes, from decode rows to prefill, and for extreme aspect ratios: what
    the cost model picks exists, has at least one k-block per split, and fits the grid."""
    rng = random.Random(5)
    log = lambda lo, hi: max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))  # noqa: E731
    shapes = [(log(1, 4096), 8 * log(32, 1792), 8 * log(32, 1792)) for _ in range(20000)]
    shapes += [(log(1, 4700000), 8 * log(1, 64), 8 * log(1, 8192)) for _ in range(5000)] + [(m, 8, 8) for m in (1, 4700000)]
    seen = set()
    for m, n, k in shapes:
        c = choice(m, n, k)
        seen.add(c)
        if c[0]:
            assert c in CONFIGS and c[2] <= -(-k // 64) and -(-m // c[0]) <= 65535, (m, n, k, c)
    assert (0, 0, 0, 0) in seen and len(seen) > 40


def _run(a, bt, out, cfg, swiglu):
    g = L.GemmArgs(a.data_ptr(), bt.data_ptr(), out.data_ptr(), 0, a.shape[0], bt.shape[0], a.shape[1], a.stride(0),
                   bt.stride(0), out.stride(0), swiglu)
    f = L.FewRows(*cfg)
    return L.lib().tccl_gemm_few_rows(C.byref(g), C.byref(f), C.c_void_p(torch.cuda.current_stream().cuda_stream))


def test_configurations_that_do_not_exist_are_refused():
    a = torch.zeros(16, 128, dtype=torch.bfloat16)
    a = a if a.data_ptr() % 16 == 0 else a.clone()
    for cfg in [(16, 2, 1, 1), (256, 1, 1, 1), (256, 2, 1, 2), (48, 1, 1, 1), (16, 1, 3, 1), (16, 1, 4, 1), (64, 2, 8, 1),
                (16, 1, 0, 1), (16, 1, 1, 0), (16, 1, 1, 3)]:  # K = 128 has two k-blocks: no split by four
        g = L.GemmArgs(a.data_ptr(), a.data_ptr(), a.data_ptr(), 0, 16, 16, 128, 128, 128, 128, 0)
        rc = L.lib().tccl_gemm_few_rows(C.byref(g), C.byref(L.FewRows(*cfg)), None)
        assert rc == -L.K["TCCL_ESIZE"], cfg


@pytest.mark.gpu
@pytest.mark.parametrize("swiglu", [0, 1])
@pytest.mark.parametrize("cfg", CONFIGS, ids=lambda c: "x".join(map(str, c)))
def test_every_configuration(cfg, swiglu):
    """Ragged edges of the tile in every direction: rows around a multiple of the token tile, columns that end inside a
    tile of Bt rows, a last k-block of 8, splits of one k-block each.  Nothing is written beside the result."""
    tn, cg, splits, _ = cfg
    gen = torch.Generator(device="cuda").manual_seed(tn * 100 + splits * 10 + cg)
    ks = (64 * splits - 56, 64 * (2 * splits + 1) + 8)
    ns = (256, 768) if swiglu else (8, 136, 264)
    for M, N, K in itertools.product((1, tn - 1, tn, 2 * tn + 3), ns, ks):
        a = torch.randn(M, K, generator=gen, device="cuda").to(torch.bfloat16)
        bt = (torch.randn(N, K, generator=gen, device="cuda") * 0.05).to(torch.bfloat16)
        cols = N // 2 if swiglu else N
        full = torch.full((M + 2, cols + 16), 77.0, dtype=torch.bfloat16, device="cuda")
        out = full[1: M + 1, 8: cols + 8]
        assert _run(a, bt, out, cfg, swiglu) == 0
        ref = a.float() @ bt.float().t()
        sums = 1e-3 * (K ** 0.5) * 0.05  # fp32 sums of K products of N(0, 1) and N(0, 0.05) in another order
        if swiglu:  # rows of Bt: blocks of 128 gate rows and the 128 matching up rows
            gr, ur = (t.reshape(M, -1) for t in ref.view(M, -1, 2, 128).unbind(2))
            ref = torch.nn.functional.silu(gr) * ur
            # |d silu| <= 1.1 |d g|: the sums' error enters through both factors; __expf adds a few units of fp32
            bound = ref.abs() * (2 ** -8 + 1e-5) + sums * (1.1 * ur.abs() + gr.abs() + 1e-3)
        else:
            bound = ref.abs() * 2 ** -8 + sums
        err = (out.float() - ref).abs()
        assert bool((err <= bound).all()), f"{(M, N, K)}: worst ratio {(err / bound).max().item()}"
        full[1: M + 1, 8: cols + 8] = 77.0
        assert bool((full == 77.0).all()), (M, N, K)


@pytest.mark.gpu
@pytest.mark.parametrize("grid", [2, 6, 20, 148])
@pytest.mark.parametrize("M,N,K", [(1024, 768, 200), (1000, 1280, 64), (1920, 2304, 136)])
def test_swiglu_half_tiles_of_the_pair_kernel(M, N, K, grid):
    """The persistent pair kernel's last partial wave: a half tile holds 64 gate columns and the 64 matching up columns."""
    gen = torch.Generator(device="cuda").manual_seed(M + N + grid)
    a = torch.randn(M, K, generator=gen, device="cuda").to(torch.bfloat16)
    bt = (torch.randn(N, K, generator=gen, device="cuda") * 0.05).to(torch.bfloat16)
    full = torch.full((M + 2, N // 2 + 16), 77.0, dtype=torch.bfloat16, device="cuda")
    out = full[1: M + 1, 8: N // 2 + 8]
    g = L.GemmArgs(a.data_ptr(), bt.data_ptr(), out.data_ptr(), 0, M, N, K, K, K, out.stride(0), 1)
    assert L.lib().tccl_gemm_bf16_pair(C.byref(g), grid, C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    gr, ur = (t.reshape(M, -1) for t in (a.float() @ bt.float().t()).view(M, -1, 2, 128).unbind(2))
    ref = torch.nn.functional.silu(gr) * ur
    bound = ref.abs() * (2 ** -8 + 1e-5) + 1e-3 * (K ** 0.5) * 0.05 * (1.1 * ur.abs() + gr.abs() + 1e-3)  # as above
    err = (out.float() - ref).abs()
    assert bool((err <= bound).all()), f"worst ratio {(err / bound).max().item()}"
    full[1: M + 1, 8: N // 2 + 8] = 77.0
    assert bool((full == 77.0).all())
