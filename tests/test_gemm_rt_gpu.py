"""The exact mode's products at the edges of their tiles: every row of a batch must carry the bits it has alone (the order of a sum
depends on its length only), whichever tile its batch took."""
import numpy as np
import pytest

import helix_b200 as hb
from helix_b200 import engine as E

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff", [(64, 128), (68, 64), (100, 36), (260, 516), (1024, 4096)])
def test_rows_do_not_depend_on_the_batch(width, ff):
    vocab = 132
    d = E.StackDesc(width=width, vocab=vocab, compute_f32=1, norm_eps=1e-6, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1,
                    layers=[E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=4, vdim=4, dim=4, kv_heads=1, norm_groups=1, conv_taps=1, ff_kind=E.FF_RELU2, ff=ff)])
    rng = np.random.default_rng(width)
    prompts = [rng.integers(0, vocab, n).tolist() for n in (1, 2, 5, 9, 33, 64, 65, 130)]
    with hb.Engine(hb.EngineConfig(max_seqs=8, max_ctx=192, max_batched_tokens=512, kv_pool_tokens=8 * 192)) as e:
        e.load_random(d, 3)
        feed = lambda batch: [(e.seq_open(), p, list(range(len(p)))) for p in batch]  # noqa: E731
        whole = feed(prompts)
        together = e.seq_step(whole)
        for s, _, _ in whole:
            e.seq_close(s)
        assert np.isfinite(together).all()
        at = 0
        for p in prompts:  # alone: 1, 2, 5 .. rows take the other tiles
            one = feed([p])
            alone = e.seq_step(one)
            e.seq_close(one[0][0])
            assert np.array_equal(alone, together[at:at + len(p)]), len(p)
            at += len(p)
