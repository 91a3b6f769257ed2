"""Quantized product with the norm in front of it in the same launch, on both sides of the line between every CTA norming for itself and the distributed form: results and the
activation left in the workspace are those of a norm kernel and the product behind it."""
import ctypes as C

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


class Mat(C.Structure):
    _fields_ = [("type", C.c_int32), ("pad", C.c_int32), ("W", C.c_void_p), ("n", C.c_int64), ("y", C.c_void_p), ("add", C.c_void_p)]


@pytest.mark.parametrize("K", [256, 512, 2304, 3840, 4096, 8192])
@pytest.mark.parametrize("types,Ns", [((O.Q4_K,), (1000,)), ((O.Q4_K, O.Q4_K, O.Q6_K), (512, 128, 96)), ((O.Q6_K,), (3,))])
def test_norm_and_product(cuda, lib, K, types, Ns):
    import torch
    ptr = lambda t: None if t is None else C.c_void_p(t.data_ptr())   # noqa: E731
    Ws = [torch.cat([torch.from_numpy(np.ascontiguousarray(O.synth_blocks(t, n, K, seed=11 + i)).reshape(-1).view(np.uint8)), torch.zeros(64, dtype=torch.uint8)]).cuda()
          for i, (t, n) in enumerate(zip(types, Ns))]
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = 3.0 * torch.randn(K, generator=g, device="cuda"), torch.rand(K, generator=g, device="cuda") + 0.5
    x[7] = 0.0
    got = []
    for sync in (torch.zeros(16, dtype=torch.uint8, device="cuda"), None):   # one launch; a norm kernel in front
        ws = torch.zeros(lib.c.pb200_act_workspace_bytes(K) + 64, dtype=torch.uint8, device="cuda")
        ys = [torch.full((n,), float("nan"), device="cuda") for n in Ns]
        mats = (Mat * len(types))(*[Mat(t, 0, W.data_ptr(), n, y.data_ptr(), None) for t, W, n, y in zip(types, Ws, Ns, ys)])
        lib.check(lib.c.pb200_gemv_fused(len(types), mats, C.c_int64(K), ptr(ws), 1, ptr(x), ptr(w), C.c_float(1e-5), ptr(sync), 0, None), "gemv_fused")
        torch.cuda.synchronize()
        got.append((ys, ws[:K]))
    assert torch.equal(got[0][1], got[1][1]) and bool((got[0][1] != 0).any())
    assert all(torch.equal(a, b) and bool(torch.isfinite(a).all()) for a, b in zip(got[0][0], got[1][0]))


# y over the vector or over the norm's weight: in place, over its end, over its start, two matrices of which the second one lies there
@pytest.mark.parametrize("K", [2048, 3840, 4096])
@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("N,at", [(4096, 0), (300, 0), (4096, 2044), (5000, -600)])
def test_result_over_an_operand(cuda, lib, K, over, N, at):
    import torch
    ptr = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    Ws = [torch.from_numpy(np.ascontiguousarray(O.synth_blocks(O.Q4_K, n, K, seed=n)).reshape(-1).view(np.uint8)).cuda() for n in (64, N)]
    buf = torch.zeros(5 * 4096, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(N + K)
    ops = [3.0 * torch.randn(K, generator=g, device="cuda"), torch.rand(K, generator=g, device="cuda") + 0.5]
    buf[8192:8192 + K] = ops[over]
    ops[over] = buf[8192:8192 + K]
    ws, sync = torch.zeros(lib.c.pb200_act_workspace_bytes(K) + 64, dtype=torch.uint8, device="cuda"), torch.zeros(16, dtype=torch.uint8, device="cuda")
    got = []
    for ys in ((torch.empty(64, device="cuda"), torch.empty(N, device="cuda")), (torch.empty(64, device="cuda"), buf[8192 + at:8192 + at + N])):
        mats = (Mat * 2)(*[Mat(O.Q4_K, 0, W.data_ptr(), y.numel(), y.data_ptr(), None) for W, y in zip(Ws, ys)])
        lib.check(lib.c.pb200_gemv_fused(2, mats, C.c_int64(K), ptr(ws), 1, ptr(ops[0]), ptr(ops[1]), C.c_float(1e-5), ptr(sync), 0, None), "gemv_fused")
        torch.cuda.synchronize()
        got.append(ys)
    assert all(torch.equal(a, b) for a, b in zip(*got))


# a programmatic launch reads neither operand before the kernel in front, a product that wrote it just now, has ended
@pytest.mark.parametrize("K", [2048, 3840, 4096])
@pytest.mark.parametrize("made", [0, 1])
def test_operand_from_the_kernel_in_front(cuda, lib, K, made):
    import torch
    ptr = lambda t: C.c_void_p(t.data_ptr())   # noqa: E731
    blocks = lambda n, k, seed: torch.from_numpy(np.ascontiguousarray(O.synth_blocks(O.Q4_K, n, k, seed=seed)).reshape(-1).view(np.uint8)).cuda()   # noqa: E731
    Kin = 8192                                       # the kernel in front takes a while
    W0, W1 = blocks(K, Kin, 3), blocks(500, K, 4)
    space = lambda k: torch.zeros(lib.c.pb200_act_workspace_bytes(k) + 64, dtype=torch.uint8, device="cuda")   # noqa: E731
    ws0, ws1, sync = space(Kin), space(K), torch.zeros(16, dtype=torch.uint8, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(K)
    xs = [torch.randn(Kin, generator=g, device="cuda") for _ in range(12)]
    other, mid = torch.rand(K, generator=g, device="cuda") + 0.5, torch.empty(K, device="cuda")

    def step(x, y, together):
        lib.check(lib.c.pb200_quantize_act(O.Q4_K, ptr(x), C.c_int64(Kin), ptr(ws0), None), "quantize_act")
        m0 = (Mat * 1)(Mat(O.Q4_K, 0, W0.data_ptr(), K, mid.data_ptr(), None))
        lib.check(lib.c.pb200_gemv_fused(1, m0, C.c_int64(Kin), ptr(ws0), 0, None, None, C.c_float(0.0), None, 1, None), "gemv_fused")
        if not together:
            torch.cuda.synchronize()
        m1 = (Mat * 1)(Mat(O.Q4_K, 0, W1.data_ptr(), 500, y.data_ptr(), None))
        in0, in1 = (mid, other) if made == 0 else (other, mid)
        lib.check(lib.c.pb200_gemv_fused(1, m1, C.c_int64(K), ptr(ws1), 1, ptr(in0), ptr(in1), C.c_float(1e-5), ptr(sync), 1 if together else 0, None), "gemv_fused")

    got, want = torch.empty(len(xs), 500, device="cuda"), torch.empty(len(xs), 500, device="cuda")
    for out, together in ((want, False), (got, True)):
        for x, y in zip(xs, out):
            step(x, y, together)
        torch.cuda.synchronize()
    assert bool(torch.isfinite(want).all()) and torch.equal(got, want)
