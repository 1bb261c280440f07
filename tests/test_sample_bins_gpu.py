"""Filtered sampling over bins of values (rows above 8192 columns): a row of 8192 columns and the same row with -inf behind it draw the same tokens,
the first by passes over the keys in one block, the second by bins in a cluster: thresholds in the bulk, values on a coarse grid (bins of hundreds
of equal logits, brackets that overflow), maxima too large for bins, temperatures whose mass ends inside or far beyond them, more survivors of
top_k than a list holds, NaN and infinities."""
import pytest
import torch

import helix_b200 as hb

pytestmark = pytest.mark.gpu


def rows(kind, B, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((B, 8192), generator=g, device="cuda") * 2
    x[:, :40] += 6
    if kind == "grid":
        x = (x * 4).round() / 4
    elif kind == "equal":
        x = torch.where(x > 1.0, 1.0, x)  # about 2500 tokens share the maximum
    elif kind == "far":
        x += 1e5
    elif kind == "beyond":
        x = x * 1e4 + 3e6
    elif kind == "nan":
        x[:, ::3] = float("nan")
    elif kind == "inf":
        x[:, 5::7] = -float("inf")
        x[::2, 11] = float("inf")
    return x


@pytest.mark.parametrize("kind", ["bulk", "grid", "equal", "far", "beyond", "nan", "inf"])
@pytest.mark.parametrize("V", [8196, 16384, 40003])
def test_bins_draw_what_keys_draw(kind, V):
    L = hb.lib()
    f = lambda v, t: torch.tensor(v, device="cuda", dtype=t)  # noqa: E731
    filters = [(t, k, p) for t in (0.05, 0.7, 1.0, 4.0) for k, p in ((0, 0.95), (0, 0.5), (0, 0.9999), (40, 0.9), (1500, 0.8), (5000, 1.0), (7, 1.0), (0, 1e-6))]
    B = len(filters)
    x = rows(kind, B, V)
    wide = torch.full((B, V), -float("inf"), device="cuda")
    wide[:, :8192] = x
    temp, tk, tp = (f([q[i] for q in filters], t) for i, t in ((0, torch.float32), (1, torch.int32), (2, torch.float32)))
    out = [torch.full((B,), -1, device="cuda", dtype=torch.int32) for _ in range(2)]
    for s in range(6):
        seed = torch.arange(B, device="cuda", dtype=torch.int64) * 7877 + s
        for o, r in zip(out, (x, wide)):
            assert L.hbk_sample_filtered(r.data_ptr(), r.shape[1], temp.data_ptr(), seed.data_ptr(), tk.data_ptr(), tp.data_ptr(), o.data_ptr(), B, r.shape[1]) == 0
        torch.cuda.synchronize()
        assert torch.equal(out[0], out[1]), (s, [filters[i] for i in (out[0] != out[1]).nonzero().flatten().tolist()])
        assert (out[0] >= 0).all()


@pytest.mark.parametrize("B", [4, 60, 130, 250])  # eight, four, two blocks and one per row
def test_more_survivors_than_a_list_holds(B):
    """top_k beyond a list's 1024 tokens together with top_p: the bins are asked twice, first for both thresholds and, since that is too many tokens, for
    the k-th alone.  The second question must not reach threads that still read the answer to the first."""
    L, V = hb.lib(), 16384
    f = lambda v, t: torch.tensor(v, device="cuda", dtype=t)  # noqa: E731
    filters = [(t, k, p) for k in (1025, 1500, 3000, 8000) for t in (0.7, 4.0) for p in (0.3, 0.8, 0.99)]
    x = rows("bulk", B, B)
    wide = torch.full((B, V), -float("inf"), device="cuda")
    wide[:, :8192] = x
    temp, tk, tp = (f([filters[b % len(filters)][i] for b in range(B)], t) for i, t in ((0, torch.float32), (1, torch.int32), (2, torch.float32)))
    out = [torch.full((B,), -1, device="cuda", dtype=torch.int32) for _ in range(2)]
    for s in range(30):
        seed = torch.arange(B, device="cuda", dtype=torch.int64) * 7877 + s
        for o, r in zip(out, (x, wide)):
            assert L.hbk_sample_filtered(r.data_ptr(), r.shape[1], temp.data_ptr(), seed.data_ptr(), tk.data_ptr(), tp.data_ptr(), o.data_ptr(), B, r.shape[1]) == 0
        torch.cuda.synchronize()
        assert torch.equal(out[0], out[1]), s


@pytest.mark.parametrize("kind", ["bulk", "grid", "equal", "far", "nan", "inf"])
@pytest.mark.parametrize("V", [8200, 32768])
def test_cold_rows(kind, V):
    """Nuclei of cold rows (bins for ten temperatures only, below 0.45): inside the bins, at their end, far below them."""
    L = hb.lib()
    f = lambda v, t: torch.tensor(v, device="cuda", dtype=t)  # noqa: E731
    filters = [(t, p) for t in (0.02, 0.1, 0.3, 0.449, 0.45) for p in (0.3, 0.9, 0.9999, 0.99999, 0.9999999)]
    B = len(filters)
    x = rows(kind, B, V)
    x[1::2, :40] -= 5  # (every other row without tokens that stand out)
    wide = torch.full((B, V), -float("inf"), device="cuda")
    wide[:, :8192] = x
    temp, tp = (f([q[i] for q in filters], torch.float32) for i in (0, 1))
    out = [torch.full((B,), -1, device="cuda", dtype=torch.int32) for _ in range(2)]
    for s in range(10):
        seed = torch.arange(B, device="cuda", dtype=torch.int64) * 7877 + s
        for o, r in zip(out, (x, wide)):
            assert L.hbk_sample_filtered(r.data_ptr(), r.shape[1], temp.data_ptr(), seed.data_ptr(), None, tp.data_ptr(), o.data_ptr(), B, r.shape[1]) == 0
        torch.cuda.synchronize()
        assert torch.equal(out[0], out[1]), (s, [filters[i] for i in (out[0] != out[1]).nonzero().flatten().tolist()])
