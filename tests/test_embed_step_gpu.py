"""The start of a stack with parallel sublayers in one launch: embedding row, its norm and both normed inputs of the first layer, against the three launches it stands
for (the same bits) and against float64.  Widths of one, two, four and eight vectors a thread, whole and with a ragged end."""
import numpy as np
import pytest
import torch

import helix_b200 as hb

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("W", [8, 1000, 1024, 1032, 2048, 3000, 4096, 4104, 8192])
@pytest.mark.parametrize("f32", [0, 1])
@pytest.mark.parametrize("pairs,off,second", [(0, 0.0, 1), (1, 1.0, 1), (1, 0.0, 0)])
def test_one_launch_equals_three(W, f32, pairs, off, second):
    l = hb.lib()
    assert l.hbk_init() == 0
    T, V, buckets, mp, mc, eps, scale = 37, 50, 11, 7919, 104729, 1e-5, 1.5
    g = torch.Generator(device="cuda").manual_seed(W + f32)
    dt = torch.float32 if f32 else BF
    table, rows = torch.randn(V, W, generator=g, device="cuda").to(dt), torch.randn(buckets + 1, W, generator=g, device="cuda").to(dt)
    w0, w1, w2 = (torch.randn(W, generator=g, device="cuda").mul(0.1).add(1.0).to(dt) for _ in range(3))
    tok = torch.randint(0, V, (T,), generator=g, device="cuda", dtype=torch.int32)
    prev = torch.randint(-1, V, (T,), generator=g, device="cuda", dtype=torch.int32)
    got = []
    for parts in (0, 1):
        x, h1, h2 = (torch.full((T, W), float("nan"), device="cuda") for _ in range(3))
        b1, b2 = (torch.full((T, W), float("nan"), device="cuda", dtype=BF) for _ in range(2))
        assert l.hbk_embed_step(tok.data_ptr(), table.data_ptr(), scale, rows.data_ptr() if pairs else None, prev.data_ptr(), buckets, mp, mc, w0.data_ptr(), off,
                                w1.data_ptr(), w2.data_ptr() if second else None, f32, eps, x.data_ptr(), h1.data_ptr(), b1.data_ptr(),
                                h2.data_ptr() if second else None, b2.data_ptr() if second else None, T, W, parts) == 0
        torch.cuda.synchronize()
        got.append((x, h1, b1) + ((h2, b2) if second else ()))
    for one, three in zip(*got):
        assert torch.isfinite(one.float()).all() and torch.equal(one, three)
    v = table[tok.long()].double() * scale
    if pairs:
        p, t = prev.cpu().numpy().astype(np.int64), tok.cpu().numpy().astype(np.int64)
        at = np.where(p < 0, buckets, (p * mp + t * mc) % buckets)
        v = v + rows[torch.from_numpy(at).cuda()].double()
    norm = lambda a, w: a / (a.square().mean(-1, keepdim=True) + eps).sqrt() * w.double()
    x = norm(v, w0.double() + off)
    # fp32: sums of up to 8192 squares (each lane a few, then 8 levels: 2^-24 * 16) and a handful of roundings, of values below 16; bf16 copies 2^-9 of theirs
    for a, want in zip(got[0], (x, norm(x, w1), norm(x, w1), norm(x, w2), norm(x, w2))):
        assert ((a.double() - want).abs() <= 2.0 ** -19 * 16 + (2.0 ** -8 if a.dtype == BF else 0.0) * want.abs()).all()


def test_rows_that_it_does_not_take():
    l = hb.lib()
    assert l.hbk_init() == 0
    buf = torch.zeros(4096, device="cuda")
    p = buf.data_ptr()
    for W, table in ((12, p), (8200, p), (64, p + 4)):
        assert l.hbk_embed_step(p, table, 1.0, None, None, 0, 0, 0, p, 0.0, p, p, 1, 1e-5, p, p, None, p, None, 1, W, 0) != 0
