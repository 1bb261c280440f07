"""State-space steps of single tokens (convolution, its moved-on inputs and the step sizes in one launch) against the same tokens fed in
one portion: one to four taps, entries that start a sequence beside running ones, sizes of the vector path and of the plain one."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("heads,vdim,state", [(4, 32, 64), (2, 16, 8), (3, 5, 7)])
@pytest.mark.parametrize("f32", [1, 0])
def test_single_tokens_equal_portions(taps, heads, vdim, state, f32):
    width, vocab = 128, 256
    layers = [E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=vdim, dim=state, kv_heads=1, norm_groups=1, conv_taps=taps, ff_kind=E.FF_RELU2, ff=256)
              for _ in range(2)]
    d = E.StackDesc(width=width, vocab=vocab, layers=layers, compute_f32=f32, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(taps * 100 + heads)
    seqs = [rng.integers(0, vocab, n).tolist() for n in (24, 20, 9, 3)]
    with hb.Engine(hb.EngineConfig(max_seqs=8, max_ctx=64, max_batched_tokens=512, kv_pool_tokens=512)) as e:
        e.load_random(d, 5)
        ids = [e.seq_open() for _ in seqs]
        whole = e.seq_step([(s, t, list(range(len(t)))) for s, t in zip(ids, seqs)])
        for s in ids:
            e.seq_close(s)
        want = np.split(whole, np.cumsum([len(t) for t in seqs])[:-1])
        ids, got = [e.seq_open() for _ in seqs], [[] for _ in seqs]
        for t in range(24):  # sequences begin at different steps, so first tokens meet running ones
            live = [i for i, s in enumerate(seqs) if 24 - len(s) <= t]
            rows = e.seq_step([(ids[i], [seqs[i][t - 24 + len(seqs[i])]], [0]) for i in live])
            for i, r in zip(live, rows):
                got[i].append(r)
        for i in range(len(seqs)):
            a, b = np.stack(got[i]).astype(np.float64), want[i].astype(np.float64)
            err = np.sqrt(((a - b) ** 2).mean(-1)) / np.sqrt((b ** 2).mean(-1))
            # two orders of summation of the same products: fp32 rounding through two layers, or bf16 roundings of inner rows that flip
            assert err.max() < (1e-5 if f32 else 3e-2), (i, err.max())
