"""-m gpu: logits of a batch step in the model's page-locked pool: the same values as through the staging buffer, arrays of their own until the last view
is gone, ordinary memory when the pool is full, life beyond the model, steps from several threads."""
import ctypes as C
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
POOL = 32 << 20
CFG = {"architecture": "Vamidra", "width": 128, "vocab": 4000, "logit_scale": 1.0, "norm": {"eps": 1e-6}, "loop": {"start": 0, "stop": 1, "times": 1},
       "layers": [{"type": "attention", "mixer": {"heads": 4, "kv_heads": 2, "dim": 32, "vdim": 32, "scale": 0.18, "softcap": 30.0, "mask": {"size": 16, "keep_first": 4}},
                   "mlp": {"kind": "dense", "ff": 256}}]}
TOKS = [np.arange(3, 3 + n, dtype=np.int32) for n in (40, 7, 1)]


def model(pkg):
    m = pkg.Model.from_config(CFG, dtype="bfloat16", n_ctx=512, n_seq=8)
    m.synth(0, 3)
    m.finalize()
    return m


def score(m, wants, into=None):
    """logits of three prompts at `wants`; into: the C call writes there instead"""
    slots = [m.seq_alloc() for _ in TOKS]
    try:
        if into is None:
            return m.batch_step([(s, t, w) for s, t, w in zip(slots, TOKS, wants)])[0]
        import importlib
        host = importlib.import_module(type(m).__module__)
        arr = (host.BatchEntry * 3)()
        ws = [np.asarray(w, dtype=np.int32) for w in wants]
        for i in range(3):
            arr[i].seq, arr[i].n_tokens, arr[i].tokens = slots[i], TOKS[i].size, TOKS[i].ctypes.data_as(C.POINTER(C.c_int32))
            arr[i].n_want, arr[i].want = ws[i].size, ws[i].ctypes.data_as(C.POINTER(C.c_int32))
        m.lib.check(m.lib.c.pb200_batch_step(m.h, 3, arr, into, None), "batch_step")
    finally:
        for s in slots:
            m.seq_free(s)


ALL = [list(range(40)), list(range(7)), [0]]


@pytest.mark.parametrize("wants", [ALL, [[39], [], [0]], [[], [6, 0, 3], []], [list(range(0, 40, 2)), [5], [0]]])
def test_same_values_wherever_they_go(cuda, pkg, wants):
    import torch
    m = model(pkg)
    rows = sum(map(len, wants))
    got = score(m, wants)
    plain = np.empty((rows, CFG["vocab"]), np.float32)
    score(m, wants, plain.ctypes.data_as(C.c_void_p))                 # ordinary memory: the staging buffer
    pinned = torch.empty(rows, CFG["vocab"]).pin_memory()
    score(m, wants, C.c_void_p(pinned.data_ptr()))                    # the caller's own page-locked memory
    assert np.isfinite(got).all() and np.array_equal(got, plain) and np.array_equal(got, pinned.numpy())
    m.close()


def test_arrays_are_their_own_until_the_last_view_is_gone(cuda, pkg):
    m = model(pkg)
    per = 48 * CFG["vocab"] * 4
    first = score(m, ALL)
    want = first.copy()
    kept = [score(m, ALL) for _ in range(POOL // per + 8)]            # more than the pool holds: the last ones lie in ordinary memory
    assert all(np.array_equal(k, want) for k in kept) and np.array_equal(first, want)
    spans = sorted((k.ctypes.data, k.nbytes) for k in kept + [first])
    assert all(a + n <= b for (a, n), (b, _) in zip(spans, spans[1:]))
    assert kept[-1].flags.owndata and not kept[0].flags.owndata
    row = kept[0][5:7]                                                # a view keeps its block
    kept.clear()
    gc.collect()
    again = [score(m, ALL) for _ in range(8)]
    assert all(not a.flags.owndata for a in again) and np.array_equal(row, want[5:7])
    m.close()
    gc.collect()
    assert np.array_equal(first, want) and all(np.array_equal(a, want) for a in again)   # blocks outlive the model
    first[:] = 1.0                                                    # and are writable


def test_blocks_come_back(cuda, pkg):
    m = model(pkg)
    take, give = m.lib.c.pb200_result_take, m.lib.c.pb200_result_give
    sizes = [1, 4096, 5000, 1 << 20, 3 << 20, 12345678]
    blocks = [take(m.h, n) for n in sizes]
    assert all(blocks) and not take(m.h, POOL) and not take(m.h, 0) and not take(None, 64)
    for b in blocks[::2] + blocks[1::2]:                              # out of order: neighbours join again
        assert give(b) == 0
    assert give(blocks[0]) == -1 and give(None) == -1 and give(blocks[0] + 64) == -1
    whole = take(m.h, POOL)
    assert whole and not take(m.h, 1) and give(whole) == 0
    m.close()


def test_steps_of_several_models_in_threads(cuda, pkg):
    ms = [model(pkg) for _ in range(3)]
    want = score(ms[0], ALL).copy()
    bad = []

    def work(m):
        held = []
        for i in range(30):
            held.append(score(m, ALL))
            if i % 3 == 2:
                held.pop(0)
        bad.extend(1 for h in held if not np.array_equal(h, want))
    ts = [threading.Thread(target=work, args=(m,)) for m in ms]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
    [m.close() for m in ms]
