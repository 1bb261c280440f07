"""Single-token steps of state-space layers in one launch between the products (heads of 128 x 64 states, four taps, a norm part per kv head): the bits
of the same tokens beside a portion, where every entry takes the kernels for portions, for 2, 4 and 8 heads per kv head, sequences that start beside
running ones, inner rows that are no whole number of blocks."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import engine as E

pytestmark = pytest.mark.gpu
VOCAB = 192


@pytest.mark.parametrize("heads,groups,ff", [(2, 1, 256), (4, 1, 1032), (8, 1, 512), (8, 2, 2056), (16, 2, 320), (4, 2, 64)])
@pytest.mark.parametrize("seqs", [1, 3, 33])
def test_single_tokens_have_the_bits_of_portions(heads, groups, ff, seqs):
    single_tokens_equal_portions(E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=64, dim=128, kv_heads=groups, norm_groups=groups, conv_taps=4, ff_kind=E.FF_RELU2, ff=ff),
                                 seqs, 4 if heads % 4 == 0 else 12)  # (with two heads the input projection's columns are no multiple of four: launches of their own)


@pytest.mark.parametrize("heads,vdim,dim,groups,norm_groups,taps", [(4, 32, 64, 2, 2, 4), (4, 64, 32, 1, 2, 3), (8, 64, 64, 2, 1, 2), (32, 64, 64, 2, 8, 4), (64, 64, 16, 8, 8, 4),
                                                                    (12, 128, 128, 3, 3, 4), (40, 36, 132, 4, 4, 1)])
@pytest.mark.parametrize("seqs", [3, 200])
def test_kernels_that_read_slabs_have_the_bits_of_portions(heads, vdim, dim, groups, norm_groups, taps, seqs):
    """Sizes that the one launch does not take: convolution and gated norm (a warp or a block per part) sum the slabs themselves, where beside a portion they read
    summed rows."""
    single_tokens_equal_portions(E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=vdim, dim=dim, kv_heads=groups, norm_groups=norm_groups, conv_taps=taps, ff_kind=E.FF_RELU2,
                                             ff=520), seqs, 6)


def single_tokens_equal_portions(layer, seqs, per_layer):
    layers, heads = [layer] * 2, layer.heads
    d = E.StackDesc(width=128, vocab=VOCAB, layers=layers, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(heads * 100 + seqs)
    toks = rng.integers(0, VOCAB, (seqs, 9)).astype(np.int32)
    steps, got, launches = 9, [], []
    with hb.Engine(hb.EngineConfig(max_seqs=seqs + 1, max_ctx=64, max_batched_tokens=256, kv_pool_tokens=64 * (seqs + 1))) as e:
        e.load_random(d, 5)
        for beside in (False, True):
            ids, rows = [e.seq_open() for _ in range(seqs)], []
            for t in range(steps):
                live = [i for i in range(seqs) if i % 3 <= t]  # sequences begin at three different steps
                feed = [(ids[i], toks[i, t - i % 3:t - i % 3 + 1], [0]) for i in live]
                other = [e.seq_open()] if beside else []
                n0 = e.stats()["kernel_launches"]
                rows.append(e.seq_step(feed + [(s, [1, 2], []) for s in other]))
                launches.append(e.stats()["kernel_launches"] - n0)
                for s in other:
                    e.seq_close(s)
            for s in ids:
                e.seq_close(s)
            got.append(np.concatenate(rows))
    assert launches[0] == 2 * per_layer + 5 and launches[-1] > launches[0]  # (embedding; final norm, product, sum, cap)
    assert np.isfinite(got[0]).all() and np.array_equal(got[0], got[1])


@pytest.mark.parametrize("budget", [0, 40, 61, 97])
def test_steps_of_256_tokens_under_an_sm_budget(budget):
    """Products cut for fewer SMs, with more slabs than on the whole machine: a step of 256 tokens has the bits of the same portions in steps of their own."""
    layers = [E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=16, vdim=64, dim=128, kv_heads=8, norm_groups=8, conv_taps=4, ff_kind=E.FF_RELU2, ff=2048) for _ in range(2)]
    d = E.StackDesc(width=512, vocab=4096, layers=layers, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    toks = np.random.default_rng(7).integers(0, 4096, (4, 64)).astype(np.int32)
    want = list(range(64))
    with hb.Engine(hb.EngineConfig(max_seqs=8, max_ctx=64, max_batched_tokens=256, kv_pool_tokens=512, sm_budget=budget)) as e:
        e.load_random(d, 5)
        ids = [e.seq_open() for _ in range(8)]
        together = e.seq_step([(s, t, want) for s, t in zip(ids, toks)])
        alone = np.concatenate([e.seq_step([(s, t, want)]) for s, t in zip(ids[4:], toks)])
    assert np.isfinite(together).all() and np.abs(together).max() > 0 and np.array_equal(together, alone)


@pytest.mark.parametrize("width,vocab,f32,budget,seqs", [(256, 4096, 0, 0, 2), (256, 4096, 0, 20, 40), (256, 4096, 1, 0, 2), (72, 190, 0, 0, 3), (68, 190, 0, 0, 3),
                                                         (256, 100003, 0, 0, 8)])
def test_rows_that_the_head_writes_to_the_host(width, vocab, f32, budget, seqs):
    """Logits up to the pinned buffer's size (four rows per sequence, 2^20 floats) and one row more, which are copied: the same rows, bit for bit."""
    layers = [E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=4, vdim=64, dim=128, kv_heads=2, norm_groups=2, conv_taps=4, ff_kind=E.FF_RELU2, ff=1024)]
    d = E.StackDesc(width=width, vocab=vocab, layers=layers, compute_f32=f32, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    limit = min(4 * seqs, 2 ** 20 // vocab)
    toks = np.random.default_rng(11).integers(0, vocab, 256 // seqs * seqs).astype(np.int32).reshape(seqs, -1)
    n = toks.shape[1]
    rows = [(i, j) for i in range(seqs) for j in range(n)]
    got = []
    with hb.Engine(hb.EngineConfig(max_seqs=seqs, max_ctx=256, max_batched_tokens=256, kv_pool_tokens=256 * seqs, sm_budget=budget)) as e:
        e.load_random(d, 5)
        for count in (limit, limit + 1):
            ids = [e.seq_open() for _ in range(seqs)]
            asked = rows[:count]
            got.append(e.seq_step([(s, t, [j for k, j in asked if k == i]) for i, (s, t) in enumerate(zip(ids, toks))]))
            for s in ids:
                e.seq_close(s)
    assert len(got[0]) == limit and len(got[1]) == limit + 1
    assert np.isfinite(got[1]).all() and np.abs(got[1]).max() > 0 and np.array_equal(got[0], got[1][:limit])
