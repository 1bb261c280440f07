"""Row passes of state-space layers at the edges of their pieces: convolution runs of eight tokens that lie inside an entry or cross its ends,
and gated group norms whose parts take one to eight vectors of a warp, a block, or single entries."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import engine as E, weights_io
from oracle import funudra_ref as ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("taps", [1, 2, 3, 4])
def test_runs_of_eight_tokens_equal_single_runs(taps):
    """2500 tokens in one step (runs of eight) against the same sequences in portions of up to 100 (runs of one): the same bits (exact mode)."""
    l = E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=4, vdim=8, dim=8, kv_heads=2, norm_groups=2, conv_taps=taps)
    d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    rng = np.random.default_rng(taps)
    seqs = [rng.integers(0, 128, n).tolist() for n in (700, 3, 1, 813, 9, 974)]
    with hb.Engine(hb.EngineConfig(max_seqs=8, max_ctx=1024, max_batched_tokens=2560, kv_pool_tokens=8192)) as e:
        e.load_random(d, 17)
        ids = [e.seq_open() for _ in seqs]
        want = np.split(e.seq_step([(s, t, list(range(len(t)))) for s, t in zip(ids, seqs)]), np.cumsum([len(t) for t in seqs])[:-1])
        for s in ids:
            e.seq_close(s)
        for t, w in zip(seqs, want):
            s = e.seq_open()
            got = np.concatenate([e.seq_step([(s, t[i:i + 100], list(range(len(t[i:i + 100]))))]) for i in range(0, len(t), 100)])
            e.seq_close(s)
            assert np.isfinite(w).all() and np.array_equal(got, w)


@pytest.mark.parametrize("heads,vdim,groups", [(4, 9, 1), (2, 16, 2), (4, 64, 1), (3, 136, 1), (6, 86, 1), (8, 128, 1), (8, 128, 2), (8, 129, 1)])
def test_group_norm_parts(heads, vdim, groups):
    cfg = ref.random_config(width=64, vocab=96, ff=64, order=(("mamba2", False),), mamba2=ref.mamba2_cfg(heads=heads, vdim=vdim, state=8, groups=1, norm_groups=groups))
    sd = ref.random_state_dict(cfg, heads * vdim)
    desc = weights_io.desc_from_hf_config(cfg, {k: v.shape for k, v in sd.items()}, compute_f32=True)
    toks = np.random.default_rng(vdim).integers(0, 96, 21).tolist()
    want = ref.FunudraOracle(cfg, sd).forward(toks)
    with hb.Engine(hb.EngineConfig(max_seqs=1, max_ctx=64, max_batched_tokens=64, kv_pool_tokens=64)) as e:
        e.load_state_dict(desc, sd)
        got = e.seq_step([(e.seq_open(), toks, list(range(21)))])
    # the exact mode's bound of the design's tests
    assert (np.sqrt(((got - want) ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))).max() < 2e-4


@pytest.mark.parametrize("heads,vdim,groups", [(8, 64, 8), (9, 96, 8), (8, 132, 8), (16, 128, 8), (16, 256, 8), (16, 260, 8)])
def test_group_norm_parts_by_warps_and_blocks(heads, vdim, groups):
    """400 tokens in one step (a warp per part of up to 512 entries) against portions of 40 (a block per part): the same bits (exact mode)."""
    l = E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=vdim, dim=8, kv_heads=1, norm_groups=groups, conv_taps=2)
    d = E.StackDesc(width=64, vocab=128, layers=[l], compute_f32=1, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)
    toks = np.random.default_rng(vdim).integers(0, 128, 400).tolist()
    with hb.Engine(hb.EngineConfig(max_seqs=2, max_ctx=448, max_batched_tokens=448, kv_pool_tokens=896)) as e:
        e.load_random(d, 19)
        want = e.seq_step([(e.seq_open(), toks, list(range(400)))])
        s = e.seq_open()
        got = np.concatenate([e.seq_step([(s, toks[i:i + 40], list(range(40)))]) for i in range(0, 400, 40)])
    assert np.isfinite(want).all() and np.array_equal(got, want)
