"""State-space layers over portions of one to many chunks of 128 tokens, ragged ones among them, at head and state sizes from narrow to wide,
against the float64 oracle, and against the same tokens fed one by one."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import weights_io
from oracle import funudra_ref as ref

pytestmark = pytest.mark.gpu


def row_err(got, want):
    d = np.asarray(got, np.float64) - want
    return np.sqrt((d * d).mean(-1)) / np.sqrt((np.asarray(want, np.float64) ** 2).mean(-1))


@pytest.mark.parametrize("heads,vdim,state,groups", [(4, 64, 128, 2), (2, 16, 8, 1), (3, 24, 72, 3), (2, 136, 16, 1), (4, 8, 64, 4)])
@pytest.mark.parametrize("cuts", [[129], [128, 128], [200, 57], [64, 300], [513]])
def test_portions_against_the_oracle(heads, vdim, state, groups, cuts):
    cfg = ref.random_config(width=128, vocab=96, ff=128, order=(("mamba2", True), ("mamba2", False)),
                            mamba2=ref.mamba2_cfg(heads=heads, vdim=vdim, state=state, groups=groups, norm_groups=1))
    sd = ref.random_state_dict(cfg, heads + sum(cuts))
    desc = weights_io.desc_from_hf_config(cfg, {k: v.shape for k, v in sd.items()}, compute_f32=False)
    rng = np.random.default_rng(sum(cuts))
    toks = rng.integers(0, 96, sum(cuts) + 3).tolist()
    want = ref.FunudraOracle(cfg, sd).forward(toks)
    with hb.Engine(hb.EngineConfig(max_seqs=2, max_ctx=640, max_batched_tokens=640, kv_pool_tokens=1280)) as e:
        e.load_state_dict(desc, sd)
        s, out, at = e.seq_open(), [], 0
        for n in cuts + [1, 1, 1]:  # the single tokens go on from the state that the portions left
            out.append(e.seq_step([(s, toks[at:at + n], list(range(n)))]))
            at += n
    # bf16 weights and operands through two layers (the serving bound of the design's tests); a lost decay, state or token is far above
    assert row_err(np.concatenate(out), want).max() < 6e-2


def test_unequal_portions_in_one_step_equal_token_by_token():
    cfg = ref.random_config(width=128, vocab=96, ff=128, order=(("mamba2", False),), mamba2=ref.mamba2_cfg(heads=4, vdim=32, state=64, groups=2, norm_groups=2))
    sd = ref.random_state_dict(cfg, 5)
    desc = weights_io.desc_from_hf_config(cfg, {k: v.shape for k, v in sd.items()}, compute_f32=False)
    rng = np.random.default_rng(6)
    seqs = [rng.integers(0, 96, n).tolist() for n in (1, 40, 127, 128, 130, 257)]
    with hb.Engine(hb.EngineConfig(max_seqs=8, max_ctx=320, max_batched_tokens=1024, kv_pool_tokens=2560)) as e:
        e.load_state_dict(desc, sd)
        ids = [e.seq_open() for _ in seqs]
        together = np.split(e.seq_step([(i, t, list(range(len(t)))) for i, t in zip(ids, seqs)]), np.cumsum([len(t) for t in seqs])[:-1])
        for i in ids:
            e.seq_close(i)
        for t, a in zip(seqs, together):
            s = e.seq_open()
            b = np.concatenate([e.seq_step([(s, [x], [0])]) for x in t])
            e.seq_close(s)
            # the products around the recurrence differ in their order of summation: flipped bf16 roundings of one layer's inner rows
            assert row_err(a, b.astype(np.float64)).max() < 1e-2
