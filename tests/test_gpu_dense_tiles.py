"""The bf16 product's tensor-core kernels at the edges of their tiles: ragged rows, tokens and k, every token tile, uncut and cut K (parts of
unequal length), the pair kernel's tiles with one and several rounds per pair, strides wider than the matrix, bias, residual and factor."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


CASES = [(5, 128, 64), (9, 130, 72), (16, 2048, 2048), (17, 300, 200), (8, 2000, 8200), (31, 1000, 1544), (64, 129, 4096), (65, 2048, 512), (130, 256, 1160), (128, 640, 8192),
         (129, 257, 64), (200, 700, 520), (256, 256, 128), (257, 513, 72), (300, 4096, 2056), (513, 1000, 1544), (1030, 5000, 264), (1500, 16000, 136)]


@pytest.mark.parametrize("T,N,K", CASES)
@pytest.mark.parametrize("extra", [False, True])
def test_product_against_float64(lib, cuda, T, N, K, extra):
    import torch
    g = torch.Generator(device="cuda").manual_seed(T * 7 + N * 3 + K)
    lda, ldw, ldc = (K + 8, K + 16, N + 3) if extra else (K, K, N)
    A = torch.randn(T, lda, generator=g, device="cuda").bfloat16()
    W = torch.randn(N, ldw, generator=g, device="cuda").bfloat16()
    A[:, K:] = float("nan")     # between the rows: never read
    W[:, K:] = float("nan")
    out = torch.full((T, ldc), 7.0, device="cuda")
    bias = torch.randn(N, generator=g, device="cuda") if extra else None
    resid = torch.randn(T, N, generator=g, device="cuda") if extra else None
    alpha = 0.5 if extra else 1.0
    lib.check(lib.c.pb200_dense(30, ptr(A), lda, ptr(W), ldw, ptr(out), ldc, T, N, K, ptr(bias), ptr(resid), N, alpha, None), "dense")
    torch.cuda.synchronize()
    assert lib.c.pb200_aborted() == 0
    a, w = A[:, :K].double(), W[:, :K].double()
    want = alpha * (a @ w.T)
    # products of bf16 are exact; every 16 of them are added with a truncation of one unit in the last place of what is there already
    bound = (K / 16 + 16) * 2.0 ** -22 * alpha * (a.abs() @ w.abs().T)
    if extra:
        want = want + bias.double() + resid.double()
        bound = bound + 2.0 ** -22 * (want.abs() + bias.double().abs() + resid.double().abs())
    assert bool(((out[:, :N].double() - want).abs() <= bound + 1e-30).all())
    assert bool((out[:, N:] == 7.0).all())


@pytest.mark.parametrize("T,N,K", [(8, 2048, 4096), (600, 1024, 512)])
def test_residual_in_place_and_repeatable(lib, cuda, T, N, K):
    """C may be the residual, and the same call gives the same bits."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    A, W = torch.randn(T, K, generator=g, device="cuda").bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16()
    x = torch.randn(T, N, generator=g, device="cuda")
    apart, inplace = torch.empty_like(x), x.clone()
    for out, resid in ((apart, x), (inplace, inplace)):
        lib.check(lib.c.pb200_dense(30, ptr(A), K, ptr(W), K, ptr(out), N, T, N, K, None, ptr(resid), N, 1.0, None), "dense")
    torch.cuda.synchronize()
    assert torch.equal(apart, inplace)


@pytest.mark.parametrize("N,K", [(2048, 8192), (4096, 2048)])
def test_a_row_in_batches_of_other_sizes(lib, cuda, N, K):
    """The cut of K, hence the order of a row's sum, follows the number of tokens: the row keeps within the bound of float64 in every batch, and its bits do
    not follow what the other rows hold."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(N)
    A, W = torch.randn(700, K, generator=g, device="cuda").bfloat16(), torch.randn(N, K, generator=g, device="cuda").bfloat16()
    B = torch.randn(700, K, generator=g, device="cuda").bfloat16()
    B[:5] = A[:5]
    want, mass = A[:5].double() @ W.double().T, A[:5].double().abs() @ W.double().abs().T
    for T in (5, 16, 17, 64, 129, 200, 300, 512, 700):
        rows = []
        for X in (A, B):
            out = torch.empty(T, N, device="cuda")
            lib.check(lib.c.pb200_dense(30, ptr(X), K, ptr(W), K, ptr(out), N, T, N, K, None, None, 0, 1.0, None), "dense")
            rows.append(out[:5])
        torch.cuda.synchronize()
        assert torch.equal(rows[0], rows[1]), T
        assert bool(((rows[0].double() - want).abs() <= (K / 16 + 16) * 2.0 ** -22 * mass).all()), T
