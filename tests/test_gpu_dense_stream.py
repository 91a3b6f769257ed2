"""The product that streams weights through shared memory (one to four tokens of bf16): pieces of a row that end inside one, CTAs without rows, odd rows of a piece
of two, more rows than a CTA keeps sums for, rows one behind the other and apart; products by themselves on both sides of the lines between it and a warp to a row."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("N,K", [(1, 256), (147, 264), (149, 2048), (300, 2056), (297, 6144), (2048, 1000), (131, 16384), (700, 13000), (150000, 256), (40000, 2048)])
@pytest.mark.parametrize("T", [1, 2, 3, 4])
def test_product_against_float64(lib, cuda, T, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(T * 7 + N * 3 + K)
    A, W = torch.randn(T, K, generator=g, device="cuda").bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16()
    bias, resid = torch.randn(N, generator=g, device="cuda"), torch.randn(T, N, generator=g, device="cuda")
    out = torch.full((T, N + 3), 7.0, device="cuda")
    lib.check(lib.c.pb200_dense(30, ptr(A), K, ptr(W), K, ptr(out), N + 3, T, N, K, ptr(bias), ptr(resid), N, 0.5, None), "dense")
    torch.cuda.synchronize()
    assert lib.c.pb200_aborted() == 0
    want = 0.5 * (A.double() @ W.double().T)
    # exact products, fp32 sums: a lane's chain of 32, five halvings of a warp and the pieces of a row, then the bias and the residual
    bound = (32 + 5 + (K + 1023) // 1024 + 3) * 2.0 ** -24 * (0.5 * (A.double().abs() @ W.double().abs().T) + bias.double().abs() + resid.double().abs())
    assert bool(((out[:, :N].double() - want - bias.double() - resid.double()).abs() <= bound).all())
    assert bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("T", [1, 3])
def test_residual_in_place(lib, cuda, T):
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    A, W = torch.randn(T, 2048, generator=g, device="cuda").bfloat16(), torch.randn(2000, 2048, generator=g, device="cuda").bfloat16()
    x = torch.randn(T, 2000, generator=g, device="cuda")
    apart, inplace = torch.empty_like(x), x.clone()
    for out, resid in ((apart, x), (inplace, inplace)):
        lib.check(lib.c.pb200_dense(30, ptr(A), 2048, ptr(W), 2048, ptr(out), 2000, T, 2000, 2048, None, ptr(resid), 2000, 1.0, None), "dense")
    torch.cuda.synchronize()
    assert torch.equal(apart, inplace)


@pytest.mark.parametrize("T", [1, 2, 4])
def test_what_the_rows_behind_hold_stays_there(lib, cuda, T):
    """Infinities in a row reach that row's results alone, and those of a token that token's."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(6)
    A, W = torch.randn(T, 1000, generator=g, device="cuda").bfloat16(), torch.randn(599, 1000, generator=g, device="cuda").bfloat16()
    clean = torch.empty(T, 599, device="cuda")
    out = torch.empty_like(clean)
    call = lambda y: lib.check(lib.c.pb200_dense(30, ptr(A), 1000, ptr(W), 1000, ptr(y), 599, T, 599, 1000, None, None, 0, 1.0, None), "dense")   # noqa: E731
    call(clean)
    W[100, 999] = float("inf")
    call(out)
    torch.cuda.synchronize()
    keep = torch.arange(599, device="cuda") != 100
    assert torch.equal(out[:, keep], clean[:, keep]) and not bool(torch.isfinite(out[:, 100]).any())


@pytest.mark.parametrize("N,K", [(2560, 2048), (2561, 2048), (3072, 2048), (3073, 2048), (4096, 1024), (1000, 11008), (4095, 4096), (4096, 4096), (16383, 2048), (16384, 2048), (20000, 2040)])
@pytest.mark.parametrize("T", [1, 2, 3, 4])
def test_both_sides_of_the_lines(lib, cuda, T, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(T * 7 + N * 3 + K)
    A, W = torch.randn(T, K, generator=g, device="cuda").bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16()
    resid = torch.randn(T, N, generator=g, device="cuda")
    out = torch.full((T, N + 3), 7.0, device="cuda")
    lib.check(lib.c.pb200_dense(30, ptr(A), K, ptr(W), K, ptr(out), N + 3, T, N, K, None, ptr(resid), N, 1.0, None), "dense")
    torch.cuda.synchronize()
    want = A.double() @ W.double().T + resid.double()
    # exact products, fp32 sums: a lane's chain of a row alone in its warp, five halvings of a warp, the warps or pieces of a row, the residual
    bound = (K // 32 + 5 + 8 + 1) * 2.0 ** -24 * (A.double().abs() @ W.double().abs().T + resid.double().abs())
    assert bool(((out[:, :N].double() - want).abs() <= bound).all()) and bool((out[:, N:] == 7.0).all())
