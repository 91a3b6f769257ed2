"""-m gpu: a model takes page-locked memory for its results when blocks are asked for, not when it is loaded."""
import pytest

import test_gpu_result_pool as R

pytestmark = pytest.mark.gpu


def resident():
    with open("/proc/self/status") as f:
        return next(int(line.split()[1]) << 10 for line in f if line.startswith("VmRSS"))


def test_a_model_without_results_holds_no_pool(cuda, pkg):
    R.model(pkg).close()                             # what the first model of a process brings along
    before = resident()
    ms = [R.model(pkg) for _ in range(6)]
    assert resident() - before < 6 * R.POOL // 2
    slots = [(m, m.seq_alloc()) for m in ms]
    assert all(m.batch_step([(s, R.TOKS[0], [])], greedy=True)[1] for m, s in slots)
    assert resident() - before < 6 * R.POOL // 2     # nor one that is asked for tokens only
    [m.close() for m in ms]


def test_slabs_grow_with_what_is_out(cuda, pkg):
    m = R.model(pkg)
    take, give = m.lib.c.pb200_result_take, m.lib.c.pb200_result_give
    before = resident()
    for _ in range(100):                             # one block after the other: one slab
        assert give(take(m.h, 1 << 20)) == 0
    assert resident() - before < 8 << 20
    out = []
    while (b := take(m.h, 1 << 20)):
        out.append(b)
    assert len(out) == R.POOL >> 20 and len(set(out)) == len(out)      # the whole bound, block by block
    assert all(give(b) == 0 for b in out[1:])
    assert not take(m.h, R.POOL)                     # one block is still out
    half = take(m.h, R.POOL // 2)                    # idle slabs make room
    assert half and give(half) == 0 and give(out[0]) == 0
    m.close()
