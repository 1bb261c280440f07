"""Kernels with tensor memory let the next kernel start only once they hold their columns (csrc/launch.h): read from the source, since the order that goes wrong
ends in two blocks that wait for one another."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "helix_b200", "csrc")
FILES = [f for f in sorted(glob.glob(os.path.join(CSRC, "*.cu"))) if "tmem_alloc" in open(f).read()]


def kernels(text):
    """(name, body) of the __global__ functions."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__", text):
        start = text.index("{", text.index(")\n", m.end()) if ")\n" in text[m.end():m.end() + 200] else m.end())
        name = re.search(r"(\w+)\s*\(\s*const", text[m.end():])
        depth, i = 0, start
        while True:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
            if depth == 0:
                break
        yield name.group(1) if name else "", text[start:i]


def test_there_are_such_kernels():
    assert len(FILES) >= 5


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_columns_before_the_next_launch(path):
    found = 0
    for name, body in kernels(open(path).read()):
        allocs = [m.end() for m in re.finditer(r"tmem_alloc(_2sm)?\(", body)]
        signals = [m.start() for m in re.finditer(r"pdl_launch_dependents\(", body)]
        found += len(allocs)
        if allocs and signals:
            assert min(signals) > max(allocs), name
    assert found
