"""Sampling and log-probability kernels (one cluster of blocks per vocabulary row) at the sizes where a slice, a vector load or a
pass can go wrong: fewer columns than blocks, ragged slices, unaligned rows, slices beyond shared memory, ties, records wider than
one merge, rows with infinities and NaN."""
import numpy as np
import pytest
import torch

import helix_b200 as hb

pytestmark = pytest.mark.gpu
SIZES = [1, 5, 31, 1000, 16387, 128256, 400009]  # 400009 / 8 columns per block do not fit shared memory


def p(t):
    return t.data_ptr() if t is not None else None


def rows_of(V, ld, seed, B=6):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((B, ld), generator=g, device="cuda") * 2
    x[1] = x[1].round()                 # ties everywhere
    x[2, ::3] = -float("inf")
    if V > 4:
        x[3, V // 2] = float("nan")
    x[4] = 0.0                          # one value; both zeros
    x[4, ::2] = -0.0
    return x


@pytest.mark.parametrize("V,B", [(v, 6) for v in SIZES] + [(v, 130) for v in SIZES[:-1]])  # (130: records of three tokens on a block per row too)
@pytest.mark.parametrize("width", [1, 2, 3, 21, 70])
def test_logprob_records(V, width, B):
    L = hb.lib()
    ld = V + 3
    x = rows_of(V, ld, V + width, B)
    sampled = torch.tensor([(7 * b) % V for b in range(B)], device="cuda", dtype=torch.int32)
    wid = torch.tensor([width] * 5 + [0] * (B - 5), device="cuda", dtype=torch.int32)
    ids = torch.full((B, width), -7, device="cuda", dtype=torch.int32)
    lps = torch.full((B, width), 5.0, device="cuda")
    assert L.hbk_logprob_topk(p(x), ld, V, p(sampled), p(wid), p(ids), p(lps), B, width) == 0
    torch.cuda.synchronize()
    assert (ids[5:] == -7).all() and (lps[5:] == 5.0).all()
    for b in range(5):
        row = x[b, :V].cpu().double().numpy()
        lse_row = row if b != 3 else None
        order = [i for i in np.lexsort((np.arange(V), -np.where(np.isnan(row), -np.inf, row))) if not np.isnan(row[i])][:width - 1]
        got = ids[b].tolist()
        assert got[0] == int(sampled[b])
        assert got[1:1 + len(order)] == [int(i) for i in order]
        if len(order) > 0:
            assert all(i == -1 for i in got[1 + len(order):])
        if lse_row is not None and np.isfinite(row.max()):
            lse = row.max() + np.log(np.exp(row - row.max()).sum())
            want = np.array([row[i] - lse for i in [got[0]] + list(order)])
            have = lps[b, :1 + len(order)].cpu().double().numpy()
            fin = np.isfinite(want)
            # fp32 sum of V positive terms in a tree of at most V / 4096 + 20 steps, each 2^-24, and expf's 2 ulp
            np.testing.assert_allclose(have[fin], want[fin], rtol=1e-6, atol=2.0 ** -24 * (V / 4096 + 40))
            assert (have[~fin] == -np.inf).all()


@pytest.mark.parametrize("V", SIZES)
def test_greedy_and_top_k_rows(V):
    """Greedy rows take the first maximum; with top_k the survivors are those that reach the k-th largest value (ties kept)."""
    L = hb.lib()
    ld = V + 1
    x = rows_of(V, ld, 31 * V)
    B = x.shape[0]
    out = torch.empty(B, device="cuda", dtype=torch.int32)
    assert L.hbk_sample(p(x), ld, None, None, p(out), B, V) == 0
    torch.cuda.synchronize()
    rows = x[:, :V].cpu().numpy()
    for b in range(B):
        r = np.where(np.isnan(rows[b]), -np.inf, rows[b])
        assert int(out[b]) == int(r.argmax())
    temp = torch.full((B,), 0.9, device="cuda")
    for k in (1, 3, 300, 5000):
        topk = torch.full((B,), k, device="cuda", dtype=torch.int32)
        for s in range(4):
            seed = torch.arange(B, device="cuda", dtype=torch.int64) * 77 + s
            assert L.hbk_sample_filtered(p(x), ld, p(temp), p(seed), p(topk), None, p(out), B, V) == 0
            torch.cuda.synchronize()
            for b in range(B):  # (a NaN is below every number)
                kth = np.sort(np.where(np.isnan(rows[b]), -np.inf, rows[b]))[::-1][min(k, V) - 1]
                assert rows[b][int(out[b])] >= kth


@pytest.mark.parametrize("V", [5, 1000, 16387, 128256, 400009])
@pytest.mark.parametrize("top_k", [0, 6])
def test_nucleus_rows(V, top_k):
    """Five tokens carry known shares (0.4 0.25 0.2 0.1 0.05) of the mass, the rest is far below the fixed point's resolution: the set
    that top_p keeps is known, with and without top_k, and every one of its tokens turns up in a few hundred draws."""
    L = hb.lib()
    B, shares = 256, np.array([0.4, 0.25, 0.2, 0.1, 0.05])
    at = np.random.default_rng(V).permutation(V)[:5]
    row = np.full(V, -60.0)
    row[at] = np.log(shares)
    x = torch.tensor(np.tile(row, (B, 1)), device="cuda", dtype=torch.float32)
    temp = torch.ones(B, device="cuda")
    for top_p, keep in ((0.3, 1), (0.5, 2), (0.8, 3), (0.9, 4), (0.99, 5)):
        tp = torch.full((B,), top_p, device="cuda")
        tk = torch.full((B,), top_k, device="cuda", dtype=torch.int32) if top_k else None
        seed = torch.arange(B, device="cuda", dtype=torch.int64) * 1234567 + V
        out = torch.empty(B, device="cuda", dtype=torch.int32)
        assert L.hbk_sample_filtered(p(x), V, p(temp), p(seed), p(tk), p(tp), p(out), B, V) == 0
        torch.cuda.synchronize()
        assert set(out.tolist()) == set(int(i) for i in at[:keep])  # the rarest survivor: missed with probability < 0.95^256


@pytest.mark.parametrize("filtered", [False, True])
@pytest.mark.parametrize("V", [8, 1000])
def test_nan_logits_are_never_drawn(V, filtered):
    """All but three logits of every row are NaN: whatever the noise, one of the three is drawn."""
    L = hb.lib()
    B = 256
    x = torch.full((B, V), float("nan"), device="cuda")
    keep = [0, V // 2, V - 1]
    x[:, keep] = torch.tensor([0.5, -1.0, 0.0], device="cuda")
    temp = torch.full((B,), 2.0, device="cuda")
    tk = torch.full((B,), V - 1, device="cuda", dtype=torch.int32) if filtered else None
    seed = torch.arange(B, device="cuda", dtype=torch.int64) * 7919
    out = torch.empty(B, device="cuda", dtype=torch.int32)
    assert L.hbk_sample_filtered(p(x), V, p(temp), p(seed), p(tk), None, p(out), B, V) == 0
    torch.cuda.synchronize()
    assert set(out.tolist()) == set(keep)


@pytest.mark.parametrize("B,V", [(32, 32768), (33, 32768), (32, 32769), (34, 32768), (5, 32769), (4, 65537), (4, 65536), (40, 1), (40, 4095), (40, 4096), (40, 8193), (200, 1000), (3, 400009)])
def test_rows_without_filters_take_the_same_tokens_either_way(B, V):
    """Rows without filters go through two launches over chunks or, few short ones and those of filtered steps, through a cluster per row:
    the same noise and the same order of ties, so the same tokens."""
    L = hb.lib()
    x = rows_of(V, V + 1, B + V, max(B, 6))
    B = x.shape[0]
    temp = torch.tensor([0.0 if b % 3 == 0 else 0.7 for b in range(B)], device="cuda")
    seed = torch.arange(B, device="cuda", dtype=torch.int64) * 104729
    no_k, no_p = torch.zeros(B, device="cuda", dtype=torch.int32), torch.ones(B, device="cuda")
    a, b = torch.full((B,), -1, device="cuda", dtype=torch.int32), torch.full((B,), -1, device="cuda", dtype=torch.int32)
    assert L.hbk_sample(p(x), V + 1, p(temp), p(seed), p(a), B, V) == 0
    assert L.hbk_sample_filtered(p(x), V + 1, p(temp), p(seed), p(no_k), p(no_p), p(b), B, V) == 0
    torch.cuda.synchronize()
    assert torch.equal(a, b) and (a >= 0).all() and (a < V).all()


def test_no_columns_are_refused():
    L = hb.lib()
    out = torch.zeros(2, device="cuda", dtype=torch.int32)
    x = torch.zeros(2, device="cuda")
    assert L.hbk_sample(p(x), 1, None, None, p(out), 2, 0) != 0


@pytest.mark.parametrize("B,V", [(48, 8192), (48, 8193), (48, 32769), (48, 100000), (48, 100001), (48, 200001), (48, 400009), (108, 16387), (108, 50000),
                                 (108, 50001), (204, 16387), (204, 25001), (204, 128256)])
def test_many_rows_equal_few(B, V):
    """Rows beside many others are shared by one, two, four or eight blocks, beside few by eight (or one): the same tokens and the same
    alternatives, whatever the number of blocks."""
    L = hb.lib()
    width = 6
    x = rows_of(V, V + 3, 7 * V, B)
    x[:, V // 3] += 9.0
    f = lambda v, t: torch.tensor(v, device="cuda", dtype=t)  # noqa: E731
    temp, seed = f([0.8, 0.5, 1.3, 0.0] * (B // 4), torch.float32), torch.arange(B, device="cuda", dtype=torch.int64) * 15485863
    topk, topp = f([0, 40, 700, 3, 0, 5000] * (B // 6), torch.int32), f([0.95, 1.0, 0.6] * (B // 3), torch.float32)
    tok = [torch.full((B,), -1, device="cuda", dtype=torch.int32) for _ in range(2)]
    ids = [torch.full((B, width), -7, device="cuda", dtype=torch.int32) for _ in range(2)]
    lps = [torch.zeros((B, width), device="cuda") for _ in range(2)]
    wid = torch.full((B,), width, device="cuda", dtype=torch.int32)
    for k, step in ((0, B), (1, 12)):
        for r in range(0, B, step):
            at = lambda t: t[r:].data_ptr()  # noqa: E731
            assert L.hbk_sample_filtered(at(x), V + 3, at(temp), at(seed), at(topk), at(topp), at(tok[k]), step, V) == 0
            assert L.hbk_logprob_topk(at(x), V + 3, V, at(tok[k]), at(wid), at(ids[k]), at(lps[k]), step, width) == 0
    torch.cuda.synchronize()
    assert torch.equal(tok[0], tok[1]) and (tok[0] >= 0).all() and (tok[0] < V).all()
    assert torch.equal(ids[0], ids[1])
    # two orders of V positive fp32 terms in trees of at most V / 512 + 20 steps; the rest is one subtraction of values below 64
    np.testing.assert_allclose(lps[0].cpu().numpy(), lps[1].cpu().numpy(), rtol=0, atol=2.0 ** -24 * (V / 512 + 20) + 2.0 ** -17)
