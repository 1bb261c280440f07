"""How prefill attention cuts a launch (host arithmetic): heads that share a tile's rows, and the order of the items."""
import os
import random
import subprocess
import sys

import pytest

import helix_b200 as hb

SMS = 148


def plan(lens, hq, hkv, paged=0):
    r = hb.load_library().hbk_attn_prefill_plan(len(lens), sum(lens), max(lens), hq, hkv, paged, SMS)
    assert r > 0
    return r & 255, r >> 8


@pytest.mark.parametrize("n,heads", [(20, 4), (33, 2), (64, 2), (90, 1), (128, 1), (129, 4), (300, 4), (3000, 4)])
def test_short_prompts_keep_their_heads_apart(n, heads):
    """32 heads over 8: what fits a lone q tile stays one, which is through sooner than a pair."""
    assert plan([n], 32, 8) == (heads, 0) and plan([n], 32, 32) == (1, 0)


@pytest.mark.parametrize("lens,hq,hkv,heads", [
    ([500 + 4000 * (i * 7 % 16) // 15 for i in range(16)], 32, 8, 2),   # 39,996 tokens: 641 rows by four, 329 by two
    ([2000 + 9300 * (i * 5 % 6) // 5 for i in range(6)], 32, 8, 2),
    ([200 + 1600 * (i * 3 % 8) // 7 for i in range(8)], 32, 1, 16),
    ([2100, 900, 700, 300], 32, 1, 16),                                 # 263 pairs by 32 do not fit an entry
    ([300, 860, 1400, 1950, 2500, 3000], 32, 8, 4),
    ([500 + 5700 * (i * 7 % 30) // 29 for i in range(30)], 32, 8, 1),
])
def test_a_packing_does_not_cost_the_order(lens, hq, hkv, heads):
    assert plan(lens, hq, hkv) == (heads, 1)
    assert plan(lens, hq, hkv, 1)[1] == 0  # pages: never sorted


def test_launches_sorted_with_heads_apart_are_sorted_packed():
    """Up to 131,072 - 256 x sequences tokens in prompts of up to 65,280 rows fit the order with heads apart: no packing may lose it."""
    rng, seen = random.Random(5), 0
    for _ in range(4000):
        hkv = rng.choice([1, 2, 4, 8])
        hq = hkv * rng.choice([1, 2, 3, 4, 6, 8, 16, 32])
        longest = int(2 ** rng.uniform(9.7, 16))
        lens = [longest] + [rng.randint(1, longest) for _ in range(rng.randint(1, 40))]
        if longest > 65280 or sum(lens) // 256 + len(lens) > 512 or not plan(lens, hq, hq)[1]:
            continue
        heads, ordered = plan(lens, hq, hkv)
        if -(-longest * heads // 256) * len(lens) * (hq // heads) <= SMS:
            continue  # (no more items than SMs: nothing to sort)
        assert (hq // hkv) % heads == 0 and ordered and longest * heads <= 65280 and sum(lens) * heads // 256 + len(lens) <= 512, (lens, hq, hkv)
        seen += 1
    assert seen > 500


def test_no_device_is_an_error():
    """The entries answer with an error where there is no device.  (The output's address, off by 8 bytes, is refused on the host where there is one.)"""
    code = ("import helix_b200 as hb; L = hb.load_library(); "
            "a = L.hbk_attn_prefill(16, 256, 16, 256, 16, 256, 8, 256, 16, 1, 10, 10, 2, 2, 64, 1, 0.1); "
            "b = L.hbk_attn_prefill_paged(16, 256, 16, 16, 16, 1, 16, 8, 256, 16, 1, 10, 10, 2, 2, 64, 1, 0.1, 1); print(a, b)")
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0 and all(int(x) != 0 for x in r.stdout.split()), (r.returncode, r.stdout)
