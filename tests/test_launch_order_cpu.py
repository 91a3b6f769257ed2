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
WAITING = [k for k in KERNELS if re.search(r"pdl_(enter|wait)\(\)", k[3])]
# weights and tables of the model, and the batch's description, which is copied in front of the pass: no kernel of the pass writes them
CONSTANT = set("""W w wa wb wn wq wk wkv wr wuk wuv w0 w1 w2 r_w bias corr sgw gateup down sink freq v_freq freq_factors A_log dt_bias Dp decay pq f_bias lower vec mu coef
                  table slot off pos0 entry_of""".split())
ALLOC = [k for k in KERNELS if "tcgen05.alloc" in k[3]]


def test_every_kernel_is_found():
    assert len(KERNELS) > 100 and len(WAITING) > 60 and len(ALLOC) == 5


@pytest.mark.parametrize("kernel", ALLOC, ids=lambda k: k[1])
def test_successor_starts_behind_the_allocation_of_tensor_memory(kernel):
    """A successor that takes columns an SM's older CTA has yet to allocate waits for that CTA, and that CTA for the columns."""
    body = kernel[3]
    assert body.rindex("tcgen05.alloc") < body.index("pdl_trigger()") and "pdl_enter()" not in body


@pytest.mark.parametrize("kernel", WAITING, ids=lambda k: k[1])
def test_results_of_earlier_kernels_are_no_constants(kernel):
    """const __restrict__ and __ldg tell the compiler that nobody writes the data while the kernel runs; it may then load ahead of the wait."""
    taken = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", kernel[2]))
    assert taken <= CONSTANT, taken - CONSTANT
    assert "__ldg(" not in kernel[3] and "ld.global.nc" not in kernel[3]


# where a role hands memory back that an asynchronous copy fills again, behind loads into registers whose values come into use later: kernel, the end of the loads, the handing back
HANDED_BACK = [("k_mmq_tc", "kg.load(", "mbar_arrive(&ctl->raw_empty"), ("k_dense_stream", "uint4 w[RB][NC];", "fetch();"),
               ("k_attn_split", "tail[2] :", "mbar_arrive(&ctl->sc_empty")]


@pytest.mark.parametrize("name,loads,back", HANDED_BACK, ids=lambda v: v if v.startswith("k_") else "")
def test_memory_is_handed_back_behind_its_loads(name, loads, back):
    """Neither a barrier's arrival nor the next copy waits for loads of shared memory that nothing has used yet."""
    (body,) = [k[3] for k in KERNELS if k[1] == name]
    start = body.index(loads)
    assert re.search(r"\bloads_done\(|\bkg\.loaded\(", body[start:body.index(back, start)])


def test_every_fork_heeds_the_switch_for_one_stream():
    s = (CSRC / "layers.cu").read_text()
    assert s.count("CK(fork_side(m))") == s.count("two_streams(ll)") == 2 and s.count('getenv("PB200_ONE_STREAM")') == 1
