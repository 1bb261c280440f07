"""State-space portions beside other entries of their step, and behind a token that is not a number: what a sequence's rows and state
are depends neither on who shares the step nor on later tokens."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import weights_io
from oracle import funudra_ref as ref

pytestmark = pytest.mark.gpu
VOCAB = 96


def stack(seed):
    cfg = ref.random_config(width=128, vocab=VOCAB, ff=128, order=(("mamba2", True), ("mamba2", False)),
                            mamba2=ref.mamba2_cfg(heads=4, vdim=64, state=128, groups=2, norm_groups=1))
    sd = ref.random_state_dict(cfg, seed)
    return sd, weights_io.desc_from_hf_config(cfg, {k: v.shape for k, v in sd.items()}, compute_f32=False)


@pytest.mark.parametrize("others", [1, 8, 30])
def test_a_portion_does_not_depend_on_its_step(others):
    """500 tokens alone and beside decoding sequences: the same bits, also of the single tokens that go on from the state left behind
    (every step here has more than 256 tokens or wants one row, so the products take the same kernels)."""
    sd, desc = stack(3)
    rng = np.random.default_rng(others)
    toks = rng.integers(0, VOCAB, 504).tolist()
    with hb.Engine(hb.EngineConfig(max_seqs=32, max_ctx=640, max_batched_tokens=1024, kv_pool_tokens=32 * 640)) as e:
        e.load_state_dict(desc, sd)
        rest = [e.seq_open() for _ in range(others)]
        e.seq_step([(s, rng.integers(0, VOCAB, 5 + i).tolist(), []) for i, s in enumerate(rest)])
        got = []
        for beside in ([], rest):
            s = e.seq_open()
            rows = [e.seq_step([(s, toks[:500], list(range(500)))] + [(o, [7], []) for o in beside])]
            rows += [e.seq_step([(s, [t], [0])]) for t in toks[500:]]
            e.seq_close(s)
            got.append(np.concatenate(rows))
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1])


def test_rows_before_a_token_that_is_not_a_number():
    sd, desc = stack(4)
    name = next(k for k, v in sd.items() if v.ndim == 2 and v.shape == (VOCAB, 128))
    sd[name] = sd[name].copy()
    sd[name][VOCAB - 1] = np.nan
    rng = np.random.default_rng(5)
    toks = rng.integers(0, VOCAB - 1, 400).tolist()
    with hb.Engine(hb.EngineConfig(max_seqs=2, max_ctx=640, max_batched_tokens=640, kv_pool_tokens=1280)) as e:
        e.load_state_dict(desc, sd)
        got = []
        for at in (None, 300):
            t = list(toks)
            if at is not None:
                t[at] = VOCAB - 1
            s = e.seq_open()
            got.append(e.seq_step([(s, t, list(range(len(t))))])[:, :VOCAB - 1])
            e.seq_close(s)
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0][:300], got[1][:300])
    assert np.isnan(got[1][300]).any()
