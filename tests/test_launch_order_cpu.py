"""Kernels that may start before the one in front has ended: what their sources have to keep to, read from the sources (no run shows a wait that a later
compiler, or another neighbour on the SM, would have needed)."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "prima.cpp_b200" / "csrc"


def kernels():
    """(file, name, signature, body) of every kernel"""
    for f in sorted(CSRC.glob("*.cu")):
        s = re.sub(r"//[^\n]*", "", f.read_text())
        for m in re.finditer(r"__global__", s):
            start = s.index("{", m.start())
            depth, i = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(s[i], 0)
                if depth == 0:
                    break
                i += 1
            sig = s[m.start():start]
            yield f.name, re.findall(r"\b(k_\w+)\(", sig)[-1], sig, s[start:i]


KERNELS = list(kernels())
ALLOC = [k for k in KERNELS if "tcgen05.alloc" in k[3]]


def test_every_kernel_is_found():
    assert len(KERNELS) > 100 and len(ALLOC) == 5


@pytest.mark.parametrize("kernel", ALLOC, ids=lambda k: k[1])
def test_successor_starts_behind_the_allocation_of_tensor_memory(kernel):
    """A successor that takes columns an SM's older CTA has yet to allocate waits for that CTA, and that CTA for the columns."""
    body = kernel[3]
    assert body.rindex("tcgen05.alloc") < body.index("pdl_trigger()") and "pdl_enter()" not in body
