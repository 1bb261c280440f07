"""Slabs of the few-token products of layer-list decoders under an SM budget: cut for fewer SMs a product can have more of them, and all that a step of 256
tokens writes has to fit what the engine sets aside."""
import ctypes as C

import pytest

import helix_b200 as hb
from helix_b200 import engine as E


def stack(width, heads, groups, ff, vocab):
    layers = [E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=heads, vdim=64, dim=128, kv_heads=groups, norm_groups=groups, conv_taps=4, ff_kind=E.FF_RELU2, ff=ff)]
    return E.StackDesc(width=width, vocab=vocab, layers=layers, norm_eps=1e-5, norm_place=E.NORM_PARALLEL, embed_norm=1, plain_gains=1, tie_head=1)


@pytest.mark.parametrize("width,heads,groups,ff,vocab", [(512, 16, 8, 2048, 4096), (512, 16, 8, 1024, 4096), (256, 8, 8, 1024, 4096), (1024, 32, 8, 4096, 4096),
                                                         (2048, 64, 8, 8192, 4096), (128, 4, 2, 512, 200)])
def test_slabs_fit_under_every_budget(width, heads, groups, ff, vocab):
    l = hb.lib()
    sd, layers = stack(width, heads, groups, ff, vocab).to_c()
    inner = heads * 64
    n_in = 2 * inner + 2 * groups * 128 + heads
    whole = l.hbk_stack_slab_floats(C.byref(sd), layers, 0)
    for budget in (0, *range(16, 149)):
        slabs = lambda n, k: l.hbk_gemm_skinny_slabs(n, k, budget or 148) * 256 * n
        have = l.hbk_stack_slab_floats(C.byref(sd), layers, budget)
        assert have >= whole
        assert slabs(n_in, width) + slabs(ff, width) <= have, budget  # two products of a launch
        assert slabs(width, inner) + slabs(width, ff) <= have, budget
        assert slabs(vocab, width) <= have, budget


def test_a_refused_description_has_no_slabs():
    l = hb.lib()
    sd, layers = stack(512, 16, 8, 1024, 4096).to_c()
    sd.width = 0
    assert l.hbk_stack_slab_floats(C.byref(sd), layers, 0) == -1
    assert l.hbk_gemm_skinny_slabs(0, 64, 16) == -1
