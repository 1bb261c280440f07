"""Prefill attention in plain order: a last round of q pairs that fills at most half of the SMs is walked as lone q tiles.  Numbers of pairs around a
half and a whole round, second tiles that are full, cut short or missing, packed keys and pages, causal or not."""
import math

import pytest
import torch

import helix_b200 as hb

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows", [128, 129, 200, 256])
@pytest.mark.parametrize("over", [(0, 1), (0, 74), (0, 75), (1, 0), (1, 1), (1, 74), (1, 75), (2, 74)])  # whole rounds and the pairs of the last one, of 148 SMs
@pytest.mark.parametrize("paged", [0, 1])
def test_last_round(D, rows, over, paged):
    L = hb.lib()
    assert L.hbk_init() == 0
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pairs = over[0] * sms + over[1] * sms // 148
    H = next(h for h in (6, 5, 4, 3, 2, 1) if pairs % h == 0)
    B, T = pairs // H, pairs // H * rows
    first = 70 if paged else 0  # positions before the first row
    causal = 1 if paged else (rows + over[1]) & 1
    g = torch.Generator(device="cuda").manual_seed(pairs + rows + D)
    qkv = torch.randn(3, T, H, D, generator=g, device="cuda").to(BF)
    out = torch.full((T, H * D), float("nan"), device="cuda", dtype=BF)
    cu = torch.arange(B + 1, device="cuda", dtype=torch.int32) * rows
    if paged:
        n = (first + rows + 63) // 64
        k, v = (torch.randn(B * n, H, 64, D, generator=g, device="cuda").to(BF) for _ in range(2))
        table = torch.arange(B * n, device="cuda", dtype=torch.int32).view(B, n).flip(0).contiguous()
        lens = torch.full((B,), first + rows, device="cuda", dtype=torch.int32)
        assert L.hbk_attn_prefill_paged(qkv[0].data_ptr(), H * D, k.data_ptr(), v.data_ptr(), table.data_ptr(), n, lens.data_ptr(), out.data_ptr(), H * D,
                                        cu.data_ptr(), B, T, rows, H, H, D, 1, D ** -0.5, B * n) == 0
        k, v = (t[table.long()].transpose(2, 3).reshape(B, n * 64, H, D)[:, :first + rows] for t in (k, v))
    else:
        assert L.hbk_attn_prefill(qkv[0].data_ptr(), H * D, qkv[1].data_ptr(), H * D, qkv[2].data_ptr(), H * D, out.data_ptr(), H * D, cu.data_ptr(), B, T,
                                  rows, H, H, D, causal, D ** -0.5) == 0
        k, v = (t.view(B, rows, H, D) for t in qkv[1:])
    torch.cuda.synchronize()
    s = torch.einsum("bnhd,bmhd->bhnm", qkv[0].view(B, rows, H, D).float(), k.float()) * D ** -0.5
    if causal:
        s.masked_fill_(torch.arange(first + rows, device="cuda")[None] > first + torch.arange(rows, device="cuda")[:, None], -math.inf)
    w = torch.einsum("bhnm,bmhd->bnhd", torch.softmax(s, -1), v.float()).reshape(T, H * D)
    # averages of unit normals: bf16 probabilities (2^-9 of a value below 5) and one bf16 rounding of the result
    assert (out.float() - w).abs().max() < 2 * 5 * 2.0 ** -9
