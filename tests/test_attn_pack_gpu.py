"""Prefill attention with the query heads of a kv head packed into a tile's rows: groups of every size (powers of two, others, single heads),
lengths around a tile's tokens for each packing, packed and paged keys, heads with gates and sinks of their own, windows, blocks and capped scores."""
import math

import pytest
import torch

import helix_b200 as hb

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def want(q, k, v, first, scale):
    """q [n, H, D], k / v [m, G, D] in fp32; query i sees the keys up to position first + i."""
    g = q.shape[1] // k.shape[1]
    s = torch.einsum("nhd,mhd->hnm", q, k.repeat_interleave(g, 1)) * scale
    at = torch.arange(k.shape[0], device=q.device)[None] > first + torch.arange(q.shape[0], device=q.device)[:, None]
    return torch.einsum("hnm,mhd->nhd", torch.softmax(s.masked_fill(at, -math.inf), -1), v.repeat_interleave(g, 1))


@pytest.mark.parametrize("Hq,Hkv", [(2, 2), (4, 2), (12, 2), (32, 8), (16, 2), (16, 1), (32, 1), (40, 1), (64, 1)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lens", [[1], [31, 32, 33], [64, 63, 65, 5], [127, 129, 257], [300, 700, 1, 513], [1100] * 4])
def test_packed_keys(Hq, Hkv, D, lens):
    L = hb.lib()
    assert L.hbk_init() == 0
    T, ld = sum(lens), (Hq + 2 * Hkv) * D
    g = torch.Generator(device="cuda").manual_seed(T + Hq)
    qkv = torch.randn(T, ld, generator=g, device="cuda").to(BF)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), device="cuda", dtype=torch.int32)
    out = torch.full((T, Hq * D), float("nan"), device="cuda", dtype=BF)
    q = qkv.data_ptr()
    assert L.hbk_attn_prefill(q, ld, q + 2 * Hq * D, ld, q + 2 * (Hq + Hkv) * D, ld, out.data_ptr(), Hq * D, cu.data_ptr(), len(lens), T, max(lens),
                              Hq, Hkv, D, 1, D ** -0.5) == 0
    torch.cuda.synchronize()
    at = 0
    for n in lens:
        x = qkv[at:at + n].float().view(n, Hq + 2 * Hkv, D)
        w = want(x[:, :Hq], x[:, Hq:Hq + Hkv], x[:, Hq + Hkv:], 0, D ** -0.5).reshape(n, -1)
        # averages of unit normals: bf16 probabilities (2^-9 of a value below 5) and one bf16 rounding of the result
        assert (out[at:at + n].float() - w).abs().max() < 2 * 5 * 2.0 ** -9
        at += n


@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (12, 2), (32, 8), (16, 1)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows,ctx", [(1, [1, 64, 300]), (33, [33, 97, 1000]), (64, [64, 2100]), (200, [300, 200, 4000]), (777, [6000]),
                                      # few rows over many keys, lone q tiles, a last kv tile that only some rows of the lower q tile see
                                      (1, [4000]), (150, [1030]), (200, [1088, 2100]), (256, [8000]), (300, [600, 520, 5000])])
def test_pages(Hq, Hkv, D, rows, ctx):
    L = hb.lib()
    assert L.hbk_init() == 0
    B, g = len(ctx), torch.Generator(device="cuda").manual_seed(rows + Hq + D)
    pages = [(c + 63) // 64 for c in ctx]
    table = torch.zeros((B, max(pages)), device="cuda", dtype=torch.int32)
    perm, at = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n] = perm[at:at + n]
        at += n
    k, v = (torch.randn((sum(pages), Hkv, 64, D), generator=g, device="cuda").to(BF) for _ in range(2))
    q = torch.randn((B * rows, Hq * D), generator=g, device="cuda").to(BF)
    out = torch.full((B * rows, Hq * D), float("nan"), device="cuda", dtype=BF)
    lens, cu = torch.tensor(ctx, device="cuda", dtype=torch.int32), torch.arange(B + 1, device="cuda", dtype=torch.int32) * rows
    assert L.hbk_attn_prefill_paged(q.data_ptr(), Hq * D, k.data_ptr(), v.data_ptr(), table.data_ptr(), table.shape[1], lens.data_ptr(), out.data_ptr(), Hq * D,
                                    cu.data_ptr(), B, B * rows, rows, Hq, Hkv, D, 1, D ** -0.5, sum(pages)) == 0
    torch.cuda.synchronize()
    for b in range(B):
        n = pages[b]
        kk, vv = (t[table[b, :n].long()].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx[b]].float() for t in (k, v))
        w = want(q[b * rows:(b + 1) * rows].float().view(rows, Hq, D), kk, vv, ctx[b] - rows, D ** -0.5).reshape(rows, -1)
        assert (out[b * rows:(b + 1) * rows].float() - w).abs().max() < 2 * 5 * 2.0 ** -9


@pytest.mark.parametrize("Hq,Hkv", [(3, 3), (12, 2), (32, 8), (16, 1)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows,ctx", [(33, [33, 97, 400]), (129, [129, 700, 1000]), (300, [300, 2100])])
@pytest.mark.parametrize("opts", [dict(window=1), dict(window=64, sink=1), dict(window=150, softcap=5.0), dict(block=50, unit=1, gate=1), dict(block=64, sink=1),
                                  dict(softcap=2.0, gate=1), dict(unit=1, sink=1, gate=1)], ids=str)
def test_what_layers_add(opts, rows, ctx, D, Hq, Hkv):
    """Windows, blocks, capped scores, sinks and gates over pages; each query head has its own sink and gates."""
    L, B = hb.lib(), len(ctx)
    assert L.hbk_init() == 0
    window, block, cap, unit = (opts.get(k, 0) for k in ("window", "block", "softcap", "unit"))
    g = torch.Generator(device="cuda").manual_seed(rows + Hq + D)
    pages = [(c + 63) // 64 for c in ctx]
    table = torch.zeros((B, max(pages)), device="cuda", dtype=torch.int32)
    perm, at = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n] = perm[at:at + n]
        at += n
    k, v = (torch.randn((sum(pages), Hkv, 64, D), generator=g, device="cuda").to(BF) for _ in range(2))
    q = torch.randn((B * rows, Hq * D), generator=g, device="cuda").to(BF)
    sink = torch.randn(Hq, generator=g, device="cuda").mul(2).to(BF) if opts.get("sink") else None
    gate = torch.randn((B * rows, Hq + 5), generator=g, device="cuda") if opts.get("gate") else None
    out, p = torch.full((B * rows, Hq * D), float("nan"), device="cuda", dtype=BF), lambda t: None if t is None else t.data_ptr()
    lens, cu = torch.tensor(ctx, device="cuda", dtype=torch.int32), torch.arange(B + 1, device="cuda", dtype=torch.int32) * rows
    assert L.hbk_attn_prefill_paged_with(p(q), Hq * D, p(k), p(v), p(table), table.shape[1], p(lens), p(out), Hq * D, p(cu), B, B * rows, rows, Hq, Hkv, D, D ** -0.5,
                                         sum(pages), window, block, cap, unit, p(sink), p(gate), Hq + 5) == 0
    torch.cuda.synchronize()
    for b in range(B):
        kk, vv = (t[table[b, :pages[b]].long()].permute(0, 2, 1, 3).reshape(-1, Hkv, D)[:ctx[b]].float().repeat_interleave(Hq // Hkv, 1) for t in (k, v))
        s = torch.einsum("nhd,mhd->hnm", q[b * rows:(b + 1) * rows].float().view(rows, Hq, D), kk) * D ** -0.5
        if cap:
            s = cap * torch.tanh(s / cap)
        i, j = torch.arange(ctx[b] - rows, ctx[b], device="cuda")[:, None], torch.arange(ctx[b], device="cuda")[None]
        seen = (j <= i) & (j > i - window if window else True) & (j >= i // block * block if block else True)
        e = torch.exp(s.masked_fill(~seen, -math.inf))
        extra = unit + (torch.exp(sink.float())[:, None, None] if sink is not None else 0)
        w = torch.einsum("hnm,mhd->nhd", e / (e.sum(-1, keepdim=True) + extra), vv)
        if gate is not None:
            w = w * torch.sigmoid(gate[b * rows:(b + 1) * rows, :Hq, None])
        # averages of unit normals: bf16 probabilities (2^-9 of a value below 5) and one bf16 rounding of the result
        assert (out[b * rows:(b + 1) * rows].float() - w.reshape(rows, -1)).abs().max() < 2 * 5 * 2.0 ** -9


@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (16, 1), (12, 2)])
def test_a_prompt_does_not_depend_on_its_launch(Hq, Hkv):
    """Alone (few items: the short ones with heads apart) and among others (packed, sorted): the same bits, also where large scores rescale the sums."""
    L, D = hb.lib(), 128
    assert L.hbk_init() == 0
    lens, ld = [90, 300, 1800, 700, 33], (Hq + 2 * Hkv) * D
    g = torch.Generator(device="cuda").manual_seed(Hq)
    qkv = (torch.randn(sum(lens), ld, generator=g, device="cuda") * 3).to(BF)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    plans = [L.hbk_attn_prefill_plan(len(ns), sum(ns), max(ns), Hq, Hkv, 0, sms) for ns in [lens] + [[n] for n in lens]]
    assert plans[0] == 256 + (Hq // Hkv & -(Hq // Hkv)) and 1 in plans
    run = []
    for at, ns in [(0, lens)] + [(sum(lens[:i]), [n]) for i, n in enumerate(lens)]:
        cu = torch.tensor([0] + list(torch.tensor(ns).cumsum(0)), device="cuda", dtype=torch.int32)
        out = torch.empty((sum(ns), Hq * D), device="cuda", dtype=BF)
        q = qkv[at:].data_ptr()
        assert L.hbk_attn_prefill(q, ld, q + 2 * Hq * D, ld, q + 2 * (Hq + Hkv) * D, ld, out.data_ptr(), Hq * D, cu.data_ptr(), len(ns), sum(ns), max(ns),
                                  Hq, Hkv, D, 1, D ** -0.5) == 0
        run.append(out)
    torch.cuda.synchronize()
    assert torch.equal(run[0], torch.cat(run[1:]))


@pytest.mark.parametrize("Hq,Hkv", [(32, 8), (16, 1), (12, 2), (4, 4)])
@pytest.mark.parametrize("D", [64, 128])
def test_a_portion_has_the_bits_of_its_prompt(Hq, Hkv, D):
    """The last rows of a prompt over its pages: alone, with a wider page table, beside other sequences, and as part of the whole prompt, the same bits."""
    L, n, ld = hb.lib(), 3000, (Hq + 2 * Hkv) * D
    assert L.hbk_init() == 0
    g = torch.Generator(device="cuda").manual_seed(Hq + D)
    qkv = (torch.randn(n, ld, generator=g, device="cuda") * 2).to(BF)
    cu, whole, p = torch.tensor([0, n], device="cuda", dtype=torch.int32), torch.empty((n, Hq * D), device="cuda", dtype=BF), qkv.data_ptr()
    assert L.hbk_attn_prefill(p, ld, p + 2 * Hq * D, ld, p + 2 * (Hq + Hkv) * D, ld, whole.data_ptr(), Hq * D, cu.data_ptr(), 1, n, n, Hq, Hkv, D, 1, D ** -0.5) == 0
    pages = (n + 63) // 64
    pool = torch.zeros((2, pages * 64, Hkv, D), device="cuda", dtype=BF)
    pool[0, :n], pool[1, :n] = (qkv[:, a:a + Hkv * D].view(n, Hkv, D) for a in (Hq * D, (Hq + Hkv) * D))
    k, v = pool.view(2, pages, 64, Hkv, D).transpose(2, 3).contiguous()
    for rows in (90, 128, 517):
        for others, width in ((0, pages), (0, 400), (2, pages), (40, pages)):
            B = 1 + others
            table = torch.arange(width, device="cuda", dtype=torch.int32).clamp(max=pages - 1).repeat(B, 1).contiguous()
            at, kv = torch.arange(B + 1, device="cuda", dtype=torch.int32) * rows, torch.full((B,), n, device="cuda", dtype=torch.int32)
            q = qkv[n - rows:, :Hq * D].repeat(B, 1).contiguous()
            out = torch.empty_like(q)
            assert L.hbk_attn_prefill_paged(q.data_ptr(), Hq * D, k.data_ptr(), v.data_ptr(), table.data_ptr(), width, kv.data_ptr(), out.data_ptr(), Hq * D, at.data_ptr(),
                                            B, B * rows, rows, Hq, Hkv, D, 1, D ** -0.5, pages) == 0
            assert torch.equal(out, whole[n - rows:].repeat(B, 1)), (rows, others, width)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (8, 2)])
def test_a_key_that_is_not_a_number_shows(Hq, Hkv, D):
    """Prompts with one NaN key at every column of two 8-column groups (each exponential has its own way): rows that see it are not finite, the others are right."""
    L, n = hb.lib(), 150
    assert L.hbk_init() == 0
    ld, at = (Hq + 2 * Hkv) * D, list(range(16)) + [63, 64, 72, 149]
    g = torch.Generator(device="cuda").manual_seed(D)
    qkv = torch.randn(len(at), n, ld, generator=g, device="cuda").to(BF)
    clean = qkv.clone()
    for b, c in enumerate(at):
        qkv[b, c, Hq * D:(Hq + Hkv) * D] = float("nan")
    cu, out = torch.arange(len(at) + 1, device="cuda", dtype=torch.int32) * n, torch.zeros((len(at), n, Hq * D), device="cuda", dtype=BF)
    q = qkv.data_ptr()
    assert L.hbk_attn_prefill(q, ld, q + 2 * Hq * D, ld, q + 2 * (Hq + Hkv) * D, ld, out.data_ptr(), Hq * D, cu.data_ptr(), len(at), len(at) * n, n, Hq, Hkv, D, 1,
                              D ** -0.5) == 0
    torch.cuda.synchronize()
    for b, c in enumerate(at):
        assert not torch.isfinite(out[b, c:].float()).any(), c
        x = clean[b].float().view(n, Hq + 2 * Hkv, D)
        w = want(x[:, :Hq], x[:, Hq:Hq + Hkv], x[:, Hq + Hkv:], 0, D ** -0.5).reshape(n, -1)
        assert (out[b, :c].float() - w[:c]).abs().max() < 2 * 5 * 2.0 ** -9 if c else True


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Hq,Hkv", [(4, 4), (8, 2)])
def test_values_behind_the_mask_have_no_weight(Hq, Hkv, D):
    """Prompts whose value rows from one position on are the largest there are: the rows before it are what they are without them."""
    L, n = hb.lib(), 150
    assert L.hbk_init() == 0
    ld, at = (Hq + 2 * Hkv) * D, list(range(1, 17)) + [63, 64, 72, 149]
    g = torch.Generator(device="cuda").manual_seed(D)
    qkv = torch.randn(n, ld, generator=g, device="cuda").to(BF).repeat(1 + len(at), 1, 1)
    for b, c in enumerate(at):
        qkv[1 + b, c:, (Hq + Hkv) * D:] = torch.finfo(BF).max
    B, out = 1 + len(at), torch.zeros((1 + len(at), n, Hq * D), device="cuda", dtype=BF)
    cu, q = torch.arange(B + 1, device="cuda", dtype=torch.int32) * n, qkv.data_ptr()
    assert L.hbk_attn_prefill(q, ld, q + 2 * Hq * D, ld, q + 2 * (Hq + Hkv) * D, ld, out.data_ptr(), Hq * D, cu.data_ptr(), B, B * n, n, Hq, Hkv, D, 1, D ** -0.5) == 0
    torch.cuda.synchronize()
    for b, c in enumerate(at):
        assert torch.equal(out[1 + b, :c], out[0, :c]), c


@pytest.mark.parametrize("D", [64, 128])
def test_encoder_rows_are_rescaled_with_their_warp(D):
    """Rows whose largest score comes in the second kv tile, up to 2^7.8 above the first's, beside one row per warp that has to be rescaled: their weight there
    is one, so the result has no rounding but its own (half a unit of 2^-7; the polynomial's 7.6e-5 in the sum of the other weights)."""
    L, n = hb.lib(), 128
    assert L.hbk_init() == 0
    qkv = torch.zeros((n, 3 * D), device="cuda", dtype=BF)
    a = torch.linspace(0.2, 5.4, n, device="cuda").to(BF)
    qkv[:, 0] = a * 8
    qkv[::32, 0], qkv[::32, 1] = 0, 16 * 8
    qkv[100, D] = qkv[101, D + 1] = 1
    qkv[100, 2 * D:] = 1
    cu, out, q = torch.tensor([0, n], device="cuda", dtype=torch.int32), torch.empty((n, D), device="cuda", dtype=BF), qkv.data_ptr()
    assert L.hbk_attn_prefill(q, 3 * D, q + 2 * D, 3 * D, q + 4 * D, 3 * D, out.data_ptr(), D, cu.data_ptr(), 1, n, n, 1, 1, D, 0, 0.125) == 0
    e = a.double().exp()
    w, rows = e / (e + n - 1), torch.arange(n, device="cuda") % 32 != 0
    assert ((out.double() - w[:, None]).abs() <= (2.0 ** (torch.floor(torch.log2(w)) - 8) + 1e-4 * w)[:, None])[rows].all()
