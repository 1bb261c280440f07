"""Every tile shape that the GEMM chooses by itself gives the bits of the narrowest one (all walk K in order) and the fp32 product, at
row counts around the edges of single tiles and of CTA pairs, ragged column counts and short K."""
import math

import pytest
import torch

import helix_b200 as hb

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
