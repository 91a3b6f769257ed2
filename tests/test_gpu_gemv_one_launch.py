"""-m gpu: pb200_mul_mat_vec in one launch (every CTA quantizes the activation) against the quantizing kernel and the product behind it: the same
integers and the same sums, so the same bits, in the result and in the caller's workspace."""
import numpy as np
import pytest
import torch

import oracle_lib as O
from gpu_util import act_ws, dev_f32, dev_u8, ptr, sync

pytestmark = pytest.mark.gpu


# one super-block, fewer than warps, a batch of loads and one more, the longest row of the one-launch way and the first one beyond it
@pytest.mark.parametrize("K,launches", [(256, 1), (1792, 1), (2048, 1), (8192, 1), (8448, 1), (14336, 1), (16384, 1), (16640, 2)])
@pytest.mark.parametrize("t", [O.Q4_K, O.Q5_K, O.Q6_K], ids=lambda t: O.TYPE_NAME[t])
@pytest.mark.parametrize("N", [1, 37, 700])
def test_one_launch_equals_two(cuda, lib, t, N, K, launches):
    x = np.random.default_rng(N + K).standard_normal(K).astype(np.float32)
    x[:256] = 0.0                                    # a super-block of zeros has the scale zero
    Wd, xd = dev_u8(O.synth_blocks(t, N, K, seed=N + K)), dev_f32(x)
    y, want, ws, ws2 = torch.full((N,), float("nan"), device="cuda"), torch.empty(N, device="cuda"), act_ws(lib, K), act_ws(lib, K)
    before = lib.c.pb200_kernel_launches()
    lib.check(lib.c.pb200_mul_mat_vec(t, ptr(Wd), N, K, ptr(xd), ptr(y), ptr(ws), None), "mul_mat_vec")
    assert lib.c.pb200_kernel_launches() - before == launches
    lib.check(lib.c.pb200_quantize_act(t, ptr(xd), K, ptr(ws2), None), "quantize_act")
    lib.check(lib.c.pb200_mul_mat_vec_q(t, ptr(Wd), N, K, ptr(ws2), ptr(want), None, None, None), "mul_mat_vec_q")
    sync()
    assert torch.equal(y, want)
    assert torch.equal(ws, ws2)


# y over x: in place, over x's end, over its start; the last ones only touch and take one launch
@pytest.mark.parametrize("N,at,launches", [(4096, 0, 2), (300, 0, 2), (4096, 4092, 2), (4096, -4092, 2), (5000, -600, 2), (4096, 4096, 1), (4096, -4096, 1)])
def test_result_over_the_activation(cuda, lib, N, at, launches):
    K, x0 = 4096, 8192
    buf = torch.zeros(5 * 4096, device="cuda")
    buf[x0:x0 + K] = torch.from_numpy(np.random.default_rng(N).standard_normal(K).astype(np.float32))
    x, y = buf[x0:x0 + K], buf[x0 + at:x0 + at + N]
    Wd, apart, ws = dev_u8(O.synth_blocks(O.Q4_K, N, K, seed=N)), torch.empty(N, device="cuda"), act_ws(lib, K)
    lib.check(lib.c.pb200_mul_mat_vec(O.Q4_K, ptr(Wd), N, K, ptr(x), ptr(apart), ptr(ws), None), "mul_mat_vec")
    before = lib.c.pb200_kernel_launches()
    lib.check(lib.c.pb200_mul_mat_vec(O.Q4_K, ptr(Wd), N, K, ptr(x), ptr(y), ptr(ws), None), "mul_mat_vec")
    assert lib.c.pb200_kernel_launches() - before == launches
    sync()
    assert torch.equal(y, apart)
