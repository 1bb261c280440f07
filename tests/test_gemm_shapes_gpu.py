"""Every tile shape that the GEMM chooses by itself gives the bits of the narrowest one (all walk K in order) and the fp32 product, at
row counts around the edges of single tiles and of CTA pairs, ragged column counts and short K."""
import math

import numpy as np
import pytest
import torch

import helix_b200 as hb
from helix_b200 import engine as E

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def rnd(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(BF)


@pytest.mark.parametrize("M", [1, 128, 129, 257, 300, 512, 513, 1281])
@pytest.mark.parametrize("N,K", [(4096, 1032), (2056, 264), (10304, 2048), (768, 3072), (136, 64)])
@pytest.mark.parametrize("epi", [0, 3, 6])  # bf16, bf16 + residual, fp32
def test_chosen_tiles(M, N, K, epi):
    l = hb.lib()
    assert l.hbk_init() == 0
    A, W, R = rnd(M, K, seed=1), rnd(N, K, scale=K ** -0.5, seed=2), rnd(M, N, seed=3)
    outs = []
    for bn in (0, 64):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32 if epi == 6 else BF)
        assert l.hbk_gemm(A.data_ptr(), K, W.data_ptr(), K, out.data_ptr(), N, R.data_ptr(), N, None, M, N, K, epi, bn) == 0
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    want = A.double() @ W.double().T + (R.double() if epi == 3 else 0)
    # fp32 sums of K products of unit variance / K (2^-24 sqrt(K) at most), then one bf16 rounding of values below 8
    bound = 2.0 ** -24 * math.sqrt(K) * 8 if epi == 6 else 8 * 2.0 ** -9 + 1e-5
    assert (outs[0].double() - want).abs().max() < bound


@pytest.mark.parametrize("M", [1, 130, 300, 520])
def test_chosen_tiles_gated(M):
    l = hb.lib()
    assert l.hbk_init() == 0
    N, K = 2048, 320
    A, W = rnd(M, K, seed=4), rnd(N, K, scale=K ** -0.5, seed=5)
    out = torch.full((M, N // 2), float("nan"), device="cuda", dtype=BF)
    assert l.hbk_gemm(A.data_ptr(), K, W.data_ptr(), K, out.data_ptr(), N // 2, None, 0, None, M, N, K, 5, 0) == 0
    torch.cuda.synchronize()
    t = (A.double() @ W.double().T).view(M, N // 256, 2, 128)
    want = (torch.nn.functional.silu(t[:, :, 0]) * t[:, :, 1]).reshape(M, -1)
    # one bf16 rounding of values below 16, the fast exponential's few ulp
    assert (out.double() - want).abs().max() < 16 * 2.0 ** -9


@pytest.mark.parametrize("M", [257, 512, 513])  # N = 4104, K = 4096: pairs of 256 x 128 below 513 rows, of 256 x 256 from there
@pytest.mark.parametrize("epi", [1, 2, 4, 10, 11])  # bias, bias + gelu, bias + residual, squared relu, gelu
def test_chosen_tiles_other_epilogues(M, epi):
    l = hb.lib()
    assert l.hbk_init() == 0
    N, K = 4104, 4096
    A, W, R, bias = rnd(M, K, seed=6), rnd(N, K, scale=K ** -0.5, seed=7), rnd(M, N, seed=8), rnd(N, seed=9)
    outs = []
    for bn in (0, 64):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=BF)
        assert l.hbk_gemm(A.data_ptr(), K, W.data_ptr(), K, out.data_ptr(), N, R.data_ptr(), N, bias.data_ptr(), M, N, K, epi, bn) == 0
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    t = A.double() @ W.double().T
    want = {1: lambda: t + bias.double(), 2: lambda: torch.nn.functional.gelu(t + bias.double()), 4: lambda: t + bias.double() + R.double(),
            10: lambda: t.clamp(min=0) ** 2, 11: lambda: torch.nn.functional.gelu(t)}[epi]()
    # one bf16 rounding of the result; fp32 sums of K products of unit variance / K behind it (2^-24 sqrt(K) times 8 at most), squared for relu^2;
    # the epilogue's erf polynomial is within 6.5e-4 of gelu (gemm.cu, gelu_erf2)
    bound = want.abs() * 2.0 ** -8 + 2.0 ** -24 * math.sqrt(K) * 8 * (2 * 8 if epi == 10 else 2) + (6.5e-4 if epi in (2, 11) else 0.0)
    assert ((outs[0].double() - want).abs() <= bound).all()


def test_silu_on_columns_gives_the_same_rows_on_every_tile():
    """The bf16 projection of linear attention with constant decays (silu on its q | k | v columns): a portion of 300 tokens alone takes pairs of
    256 x 128, beside 300 more tokens pairs of 256 x 256; its rows keep their bits."""
    l = E.LayerDesc(mixer=E.MIXER_LIGHTNING, heads=8, vdim=128, dim=128, head_decay=tuple(0.5 + 0.06 * i for i in range(8)))
    d = E.StackDesc(width=4096, vocab=128, layers=[l], norm_eps=1e-5, norm_place=E.NORM_PRE, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(1)
    toks = rng.integers(0, 128, 300).tolist()
    with hb.Engine(hb.EngineConfig(max_seqs=8, max_ctx=1024, max_batched_tokens=2048, kv_pool_tokens=8 * 1024)) as e:
        e.load_random(d, 2)
        got = []
        for beside in ([], [40], [300], [1000]):
            ids = [e.seq_open() for _ in range(1 + len(beside))]
            got.append(e.seq_step([(ids[0], toks, list(range(300)))] + [(i, rng.integers(0, 128, n).tolist(), []) for i, n in zip(ids[1:], beside)]))
            for i in ids:
                e.seq_close(i)
    assert np.isfinite(got[0]).all()
    for g in got[1:]:
        assert np.array_equal(got[0], g)


@pytest.mark.parametrize("M,N,K", [(1280, 2048, 1032), (2305, 2056, 72), (2305, 4104, 72), (1537, 1544, 1032), (2561, 2048, 64), (2305, 3976, 328)])
@pytest.mark.parametrize("epi", [0, 2, 3, 6])  # bf16, bias + gelu, bf16 + residual, fp32
def test_tiles_of_192_columns(M, N, K, epi):
    """Sizes whose waves end first in 256 x 192: whole and ragged rows and columns, a last tile of a few columns, one k block."""
    l = hb.lib()
    assert l.hbk_init() == 0
    assert tile(M, N, K, epi) == (192, 2, 4 if epi in (2, 3) and K < 1000 else 2)
    same_as_narrow_tiles(M, N, K, epi)


@pytest.mark.parametrize("M,N,K", [(3000, 3072, 768), (3000, 4104, 72), (4609, 2304, 64), (7000, 2056, 328)])
@pytest.mark.parametrize("epi", [2, 3])
def test_four_epilogue_groups_on_256_columns(M, N, K, epi):
    """Sizes that take tiles of 256 x 256 with four groups of epilogue warps: whole and ragged rows and columns, one k block and several."""
    l = hb.lib()
    assert l.hbk_init() == 0
    assert tile(M, N, K, epi) == (256, 2, 4)
    same_as_narrow_tiles(M, N, K, epi)


def tile(M, N, K, epi):
    t = hb.lib().hbk_gemm_tile(M, N, K, epi, torch.cuda.get_device_properties(0).multi_processor_count)
    return t & 4095, t >> 12 & 15, t >> 16


def same_as_narrow_tiles(M, N, K, epi):
    l = hb.lib()
    A, W, R, b = rnd(M, K, seed=6), rnd(N, K, scale=K ** -0.5, seed=7), rnd(M, N, seed=8), rnd(N, seed=9)
    outs = []
    for bn in (0, 64):
        out = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float32 if epi == 6 else BF)
        assert l.hbk_gemm(A.data_ptr(), K, W.data_ptr(), K, out.data_ptr(), N, R.data_ptr(), N, b.data_ptr(), M, N, K, epi, bn) == 0
        torch.cuda.synchronize()
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    want = A.double() @ W.double().T
    want = want + R.double() if epi == 3 else torch.nn.functional.gelu(want + b.double()) if epi == 2 else want
    # fp32 sums of K products of unit variance / K (2^-24 sqrt(K) at most), then one bf16 rounding of values below 8 (below 16 with a bias; the gelu's polynomial 6.5e-4)
    bound = 2.0 ** -24 * math.sqrt(K) * 8 if epi == 6 else 16 * 2.0 ** -9 + 1e-3
    assert (outs[0].double() - want).abs().max() < bound
