"""-m gpu: logits of a batch step into memory whose ends are page-locked by different registrations, with ordinary pages or nothing between them: one copy
cannot take such a range, the step goes through the staging buffer."""
import ctypes as C

import numpy as np
import pytest
import torch

import test_gpu_result_pool as R

pytestmark = pytest.mark.gpu
PAGE = 4096


@pytest.mark.parametrize("locked", [[(0, 40), (60, 188)], [(0, 64), (64, 188)], [(0, 1), (1, 187), (187, 188)], [(0, 188)], [(0, 100)], [(90, 188)]],
                         ids=["gap", "side by side", "three", "whole", "first half", "second half"])
def test_ranges_of_several_registrations(cuda, pkg, locked):
    m = R.model(pkg)
    want = R.score(m, R.ALL).copy()
    assert want.nbytes == 768000 and -(-want.nbytes // PAGE) == 188
    raw = np.empty(want.nbytes + 2 * PAGE, np.uint8)
    at = -raw.ctypes.data % PAGE
    rows = raw[at:at + want.nbytes].view(np.float32).reshape(want.shape)
    rows[:] = np.nan
    rt, base = torch.cuda.cudart(), raw.ctypes.data + at
    for a, b in locked:
        assert int(rt.cudaHostRegister(base + a * PAGE, (b - a) * PAGE, 0)) == 0
    try:
        R.score(m, R.ALL, C.c_void_p(base))
        assert np.array_equal(rows, want)
    finally:
        for a, _ in locked:
            assert int(rt.cudaHostUnregister(base + a * PAGE)) == 0
        m.close()
