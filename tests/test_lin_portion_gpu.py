"""Portions on the recurrence's wide kernel (no normaliser, more than 32 channels and columns): stages of 16 tokens, pairs and a single last token,
padded channels and columns, narrow and wide blocks, a state left by an earlier portion.  The exact mode's logits must equal, bit for bit,
those of the same tokens fed one at a time (another kernel, the same sums in the same order)."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["ssm", "lightning"])
@pytest.mark.parametrize("heads,dim,vdim", [(4, 36, 36), (4, 64, 64), (4, 128, 64), (40, 128, 64), (4, 72, 136), (4, 256, 40), (40, 256, 64), (40, 132, 68)])
def test_portions_equal_single_tokens(kind, heads, dim, vdim):
    if kind == "ssm":
        l = E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=vdim, dim=dim, kv_heads=2, norm_groups=1, conv_taps=1)
        d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    else:
        l = E.LayerDesc(mixer=E.MIXER_LIGHTNING, heads=heads, vdim=vdim, dim=dim, head_decay=tuple(np.linspace(0.0, 1.0, heads)))
        d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PRE, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(heads + dim + vdim)
    cuts = [(33, 18), (16, 31), (1, 40), (17, 1)]  # two portions of four sequences
    seqs = [rng.integers(0, 128, sum(c)).tolist() for c in cuts]
    with hb.Engine(hb.EngineConfig(max_seqs=4, max_ctx=64, max_batched_tokens=256, kv_pool_tokens=256)) as e:
        e.load_random(d, 13)
        ids, want = [e.seq_open() for _ in seqs], [[] for _ in seqs]
        for part in range(2):
            toks = [t[:c[0]] if part == 0 else t[c[0]:] for t, c in zip(seqs, cuts)]
            rows = e.seq_step([(s, t, list(range(len(t)))) for s, t in zip(ids, toks)])
            for w, r in zip(want, np.split(rows, np.cumsum([len(t) for t in toks])[:-1])):
                w.append(r)
        for s in ids:
            e.seq_close(s)
        ids, got = [e.seq_open() for _ in seqs], [[] for _ in seqs]
        for at in range(max(map(len, seqs))):
            live = [i for i, t in enumerate(seqs) if at < len(t)]
            for i, r in zip(live, e.seq_step([(ids[i], [seqs[i][at]], [0]) for i in live])):
                got[i].append(r)
    for a, b in zip(got, want):
        b = np.concatenate(b)
        assert np.isfinite(b).all() and np.array_equal(np.stack(a), b)


@pytest.mark.parametrize("kind", ["ssm", "lightning"])
@pytest.mark.parametrize("heads,dim,vdim", [(40, 128, 64), (40, 72, 136), (40, 256, 64), (40, 132, 68)])
def test_longer_portions_on_wide_blocks_equal_single_tokens(kind, heads, dim, vdim):
    if kind == "ssm":
        l = E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=vdim, dim=dim, kv_heads=2, norm_groups=1, conv_taps=1)
        d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    else:
        l = E.LayerDesc(mixer=E.MIXER_LIGHTNING, heads=heads, vdim=vdim, dim=dim, head_decay=tuple(np.linspace(0.0, 1.0, heads)))
        d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PRE, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(heads + dim + vdim)
    cuts = [(49, 18), (16, 33), (1, 66), (48, 1)]  # two portions of four sequences, more than 24 tokens on average
    seqs = [rng.integers(0, 128, sum(c)).tolist() for c in cuts]
    with hb.Engine(hb.EngineConfig(max_seqs=4, max_ctx=128, max_batched_tokens=256, kv_pool_tokens=512)) as e:
        e.load_random(d, 13)
        ids, want = [e.seq_open() for _ in seqs], [[] for _ in seqs]
        for part in range(2):
            toks = [t[:c[0]] if part == 0 else t[c[0]:] for t, c in zip(seqs, cuts)]
            rows = e.seq_step([(s, t, list(range(len(t)))) for s, t in zip(ids, toks)])
            for w, r in zip(want, np.split(rows, np.cumsum([len(t) for t in toks])[:-1])):
                w.append(r)
        for s in ids:
            e.seq_close(s)
        ids, got = [e.seq_open() for _ in seqs], [[] for _ in seqs]
        for at in range(max(map(len, seqs))):
            live = [i for i, t in enumerate(seqs) if at < len(t)]
            for i, r in zip(live, e.seq_step([(ids[i], [seqs[i][at]], [0]) for i in live])):
                got[i].append(r)
    for a, b in zip(got, want):
        b = np.concatenate(b)
        assert np.isfinite(b).all() and np.array_equal(np.stack(a), b)


@pytest.mark.parametrize("kind", ["ssm", "lightning"])
@pytest.mark.parametrize("heads,dim,vdim", [(120, 128, 64), (120, 68, 36)])
def test_many_blocks_equal_single_tokens(kind, heads, dim, vdim):
    """More blocks than three per SM: eight columns per lane, also with padded channels and columns."""
    test_longer_portions_on_wide_blocks_equal_single_tokens(kind, heads, dim, vdim)
