"""-m gpu: while a trace buffer is set, the single product runs instrumented too (by two launches), and takes its one launch again afterwards; a product with the norm in front of it runs
in the form that it has without the buffer."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle_lib as O
from gpu_util import act_ws, dev_f32, dev_u8, ptr, sync

pytestmark = pytest.mark.gpu


def test_single_product_is_traced(cuda, lib):
    N, K, row = 4096, 4096, 4096
    Wd, xd, y, ws = dev_u8(O.synth_blocks(O.Q4_K, N, K, seed=1)), dev_f32(np.random.default_rng(1).standard_normal(K)), torch.empty(N, device="cuda"), act_ws(lib, K)
    trace = torch.zeros(2 * row, dtype=torch.int64, device="cuda")
    set_trace = lib.c.pb200_debug_set_trace
    set_trace.argtypes = [C.c_void_p, C.c_int]

    def call():
        before = lib.c.pb200_kernel_launches()
        lib.check(lib.c.pb200_mul_mat_vec(O.Q4_K, ptr(Wd), N, K, ptr(xd), ptr(y), ptr(ws), None), "mul_mat_vec")
        sync()
        return lib.c.pb200_kernel_launches() - before, y.clone()
    n1, plain = call()
    lib.check(set_trace(ptr(trace), 2), "set_trace")
    try:
        n2, traced = call()
    finally:
        lib.check(set_trace(None, 0), "set_trace")
    n3, again = call()
    assert (n1, n2, n3) == (1, 2, 1) and torch.equal(plain, traced) and torch.equal(plain, again)
    t = trace.cpu().numpy().reshape(2, -1, 8)
    ctas = int((t[0, :, 0] != 0).sum())
    assert ctas > 100 and (t[1] == 0).all() and (np.diff(t[0, :ctas, :6], axis=1) >= 0).all()


@pytest.mark.parametrize("K", [2048, 4096])          # every CTA norms for itself, and the distributed form
def test_product_with_a_norm_is_traced(cuda, lib, K):
    from test_gpu_gemv_norm import Mat
    N, row = 3000, 4096
    Wd, ws, bar = dev_u8(O.synth_blocks(O.Q5_K, N, K, seed=2)), act_ws(lib, K), torch.zeros(16, dtype=torch.uint8, device="cuda")
    x, w = dev_f32(np.random.default_rng(2).standard_normal(K)), dev_f32(np.random.default_rng(3).random(K) + 0.5)
    trace = torch.zeros(2 * row, dtype=torch.int64, device="cuda")
    set_trace = lib.c.pb200_debug_set_trace
    set_trace.argtypes = [C.c_void_p, C.c_int]

    def call():
        y = torch.full((N,), float("nan"), device="cuda")
        mats = (Mat * 1)(Mat(O.Q5_K, 0, Wd.data_ptr(), N, y.data_ptr(), None))
        lib.check(lib.c.pb200_gemv_fused(1, mats, C.c_int64(K), ptr(ws), 1, ptr(x), ptr(w), C.c_float(1e-5), ptr(bar), 0, None), "gemv_fused")
        sync()
        return y
    plain = call()
    lib.check(set_trace(ptr(trace), 2), "set_trace")
    try:
        traced = call()
    finally:
        lib.check(set_trace(None, 0), "set_trace")
    assert torch.equal(plain, traced) and bool(torch.isfinite(plain).all())
    t = trace.cpu().numpy().reshape(2, -1, 8)
    ctas = int((t[0, :, 0] != 0).sum())
    assert ctas > 100 and (t[1] == 0).all() and (np.diff(t[0, :ctas, :6], axis=1) >= 0).all()
