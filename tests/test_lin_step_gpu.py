"""Single-token steps of the scalar-decay recurrences (state-space layers, linear attention with constant decays) at head sizes around a
warp's sixteen channels and a block's 64 columns, first tokens beside running ones: the exact mode's logits must equal, row by
row, those of the same sequences fed in portions (another kernel, the same arithmetic and fp32 products in the same order)."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ssm", "lightning"])
@pytest.mark.parametrize("dim,vdim", [(4, 2), (16, 64), (20, 66), (128, 64), (128, 130), (256, 40), (7, 5)])
def test_single_tokens(kind, dim, vdim):
    if kind == "ssm":
        l = E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=4, vdim=vdim, dim=dim, kv_heads=2, norm_groups=1, conv_taps=1)
        d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    else:
        l = E.LayerDesc(mixer=E.MIXER_LIGHTNING, heads=4, vdim=vdim, dim=dim, head_decay=(0.9, 0.5, 1.0, 0.0))
        d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PRE, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(dim + vdim)
    seqs = [rng.integers(0, 128, n).tolist() for n in (12, 7, 3)]
    with hb.Engine(hb.EngineConfig(max_seqs=4, max_ctx=64, max_batched_tokens=256, kv_pool_tokens=256)) as e:
        e.load_random(d, 11)
        ids = [e.seq_open() for _ in seqs]
        want = np.split(e.seq_step([(s, t, list(range(len(t)))) for s, t in zip(ids, seqs)]), np.cumsum([len(t) for t in seqs])[:-1])
        for s in ids:
            e.seq_close(s)
        ids, got = [e.seq_open() for _ in seqs], [[] for _ in seqs]
        for t in range(12):
            live = [i for i, s in enumerate(seqs) if 12 - len(s) <= t]
            for i, r in zip(live, e.seq_step([(ids[i], [seqs[i][t - 12 + len(seqs[i])]], [0]) for i in live])):
                got[i].append(r)
        for a, b in zip(got, want):
            assert np.array_equal(np.stack(a), b)


def test_narrow_heads_beside_thousands():
    """Heads of up to 32 columns leave the single-token kernel beside more than 4096 (sequence, head) pairs: 66 sequences x 64 heads in one step give
    the bits of the same sequences in two steps of 33."""
    l = E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=64, vdim=6, dim=8, kv_heads=4, norm_groups=1, conv_taps=1)
    d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(1)
    first, then = rng.integers(0, 128, (66, 2)).tolist(), rng.integers(0, 128, (66, 2)).tolist()
    got = []
    with hb.Engine(hb.EngineConfig(max_seqs=66, max_ctx=64, max_batched_tokens=256, kv_pool_tokens=66 * 64)) as e:
        e.load_random(d, 12)
        for parts in ([slice(0, 66)], [slice(0, 33), slice(33, 66)]):
            ids = [e.seq_open() for _ in first]
            e.seq_step([(s, t, []) for s, t in zip(ids, first)])
            rows = [np.concatenate([e.seq_step([(s, [t[k]], [0]) for s, t in zip(ids[p], then[p])]) for p in parts]) for k in range(2)]
            for s in ids:
                e.seq_close(s)
            got.append(np.stack(rows))
    assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1])
