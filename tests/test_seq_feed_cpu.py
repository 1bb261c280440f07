"""Engine.seq_step's argument forms, down to the descriptors that cross the C ABI: no GPU, the library call is a recorder."""
import ctypes as C
from types import SimpleNamespace

import numpy as np
import pytest

from helix_b200.engine import Engine


def described(entries):
    """What the library would be handed: [(id, tokens, want)]."""
    seen = []

    def hb_seq_step(h, arr, n, out, cap, got):
        for f in arr[:n]:
            toks = np.ctypeslib.as_array(C.cast(f.tokens, C.POINTER(C.c_int32)), (f.n_tokens,)).tolist() if f.n_tokens else []
            want = np.ctypeslib.as_array(C.cast(f.want, C.POINTER(C.c_int32)), (f.n_want,)).tolist() if f.n_want else []
            seen.append((f.seq, toks, want))
        return 0

    e = Engine.__new__(Engine)
    e._l, e._h, e.desc, e._ck = SimpleNamespace(hb_seq_step=hb_seq_step, hb_engine_destroy=lambda h: None), None, SimpleNamespace(vocab=3), lambda rc: None
    out = e.seq_step(entries)
    assert out.shape == (sum(len(w) for _, _, w in seen), 3)
    return seen


@pytest.mark.parametrize("sid", [0, 5, 2 ** 64 - 1, -1, 2 ** 64 + 5, np.int64(3), True])
def test_ids_wrap_as_unsigned_64(sid):
    assert described([(sid, [1], [0])]) == [(int(sid) % 2 ** 64, [1], [0])]


@pytest.mark.parametrize("sid", [3.0, "3", None])
def test_ids_that_are_no_integers(sid):
    with pytest.raises(TypeError):
        described([(sid, [1], [0])])


def test_any_sized_collection_of_triples():
    want = [(1, [4, 5], [1]), (2, [6], [])]
    by_id = {e[0]: e for e in want}
    assert described(by_id.values()) == want
    assert described(tuple(want)) == want
    assert described([list(e) for e in want]) == want

    class Triple:  # (an entry needs no more than to unpack)
        def __iter__(self):
            return iter((7, np.array([1, 2]), np.array([0, 1], np.int64)))

    assert described([Triple()]) == [(7, [1, 2], [0, 1])]
