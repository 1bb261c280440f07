"""Prefill attention at the edges of its item order: as many rows (q pairs of all sequences) as the sorted order holds and one more, as many
sequences as its entries name and one more, empty sequences among sorted ones, one row, fewer items than blocks."""
import math

import pytest
import torch

import helix_b200 as hb

pytestmark = pytest.mark.gpu
BF = torch.bfloat16

LENS = {
    "one": [1], "fewer_items_than_blocks": [300, 40], "uneven": [3, 700, 256, 257, 90, 1025, 511, 64], "empty_ones": [0, 130, 0, 600, 0],
    "rows_512": [256] * 128 + [512] * 64 + [513] * 64 + [512] * 32, "rows_513": [1] * 200 + [1800] * 39 + [129], "sequences_256": [33] * 255 + [500],
    "sequences_257": [33] * 256 + [500], "rows_512_exactly": [1] * 200 + [1800] * 39, "sequences_256_sorted": [65] * 255 + [1500],
    "sequences_257_long": [65] * 256 + [1500], "empty_ones_sorted": [0, 130, 0, 1100, 0, 900, 257, 300],
}


@pytest.mark.parametrize("name", list(LENS))
@pytest.mark.parametrize("D,Hq,Hkv,causal", [(128, 4, 2, 1), (64, 3, 3, 0), (64, 4, 1, 1)])
def test_item_order(name, D, Hq, Hkv, causal):
    l = hb.lib()
    assert l.hbk_init() == 0
    lens = LENS[name][:256] if name == "rows_512" else LENS[name]
    T = sum(lens)
    g = torch.Generator(device="cuda").manual_seed(T)
    ld = (Hq + 2 * Hkv) * D
    qkv = torch.randn(T, ld, generator=g, device="cuda").to(BF)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device="cuda", dtype=torch.int32)
    out = torch.full((T, Hq * D), float("nan"), device="cuda", dtype=BF)
    want = torch.empty(T, Hq * D, device="cuda")
    q = qkv.data_ptr()
    args = (q, ld, q + 2 * Hq * D, ld, q + 2 * (Hq + Hkv) * D, ld)
    tail = (Hq * D, cu.data_ptr(), len(lens), T, max(lens), Hq, Hkv, D, causal, 1 / math.sqrt(D))
    assert l.hbk_attn_prefill(*args, out.data_ptr(), *tail) == 0
    assert l.hbk_attn_naive(*args, want.data_ptr(), *tail) == 0
    torch.cuda.synchronize()
    # averages of unit normals: bf16 probabilities (2^-9 of a value below 5) and one bf16 rounding of the result
    assert (out.float() - want).abs().max() < 2 * 5 * 2.0 ** -9
