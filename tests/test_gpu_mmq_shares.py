"""-m gpu: the k-quant product in each of the ways its tiles are shared among CTAs.

Bound: the element-wise fp16-roundings bound and NMSE of test_gpu_mmq.check; a cut adds one fp32 rounding per CTA of the tile, far below it.
"""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_mmq import check, oracle, run_mmq

pytestmark = pytest.mark.gpu


# (rows, K, tokens): on 148 SMs K cut over 2, 4 and 8 CTAs, halves and whole tiles, shares that end inside tiles (20480 x 2048), chains of two tiles
# (11008 x 4096), and the edges of the 16-token chunks that the 16 reading warps take (1, 15, 17 tokens; a second accumulator with one token;
# rows that end inside a tile)
@pytest.mark.parametrize("N,K,T", [(200, 2048, 1), (130, 3072, 15), (128, 4096, 17), (20480, 512, 17), (3840, 2816, 257), (14336, 256, 31), (129, 1024, 513), (20480, 2048, 33), (11008, 4096, 33)])
@pytest.mark.parametrize("extra", [False, True], ids=["plain", "bias_residual"])
def test_mmq_shares(cuda, lib, port, N, K, T, extra):
    rng = np.random.default_rng(N + K + T)
    W = O.synth_blocks(O.Q4_K, N, K, seed=N + T)
    X = rng.standard_normal((T, K)).astype(np.float32)
    bias = rng.standard_normal(N).astype(np.float32) if extra else None
    resid = rng.standard_normal((T, N)).astype(np.float32) if extra else None
    got = run_mmq(lib, O.Q4_K, W, N, K, X, bias=bias, resid=resid)
    want = oracle(port, O.Q4_K, W, N, K, X)
    if extra:
        want = want + bias + resid
    check(got, want, port.dequantize(O.Q4_K, W, N * K).reshape(N, K), X)


# K cut over 8, 4, 3 and 2 CTAs of a cluster (equal and unequal parts), halves, chains of two and three tiles, contiguous shares of a tile and more, whole
# tiles; few tokens to two rounds of two accumulators; every block type
@pytest.mark.parametrize("t,N,K", [(O.Q4_K, 1024, 4096), (O.Q4_K, 4096, 4096), (O.Q5_K, 2000, 2048), (O.Q6_K, 5000, 3840), (O.Q4_K, 9000, 2560), (O.Q4_K, 11008, 4096), (O.Q4_K, 12800, 8192), (O.Q4_K, 20480, 2048),
                                   (O.Q4_K, 14336, 1024), (O.Q8_0, 1000, 2112), (O.Q5_1, 500, 1984)])
@pytest.mark.parametrize("T", [9, 260, 512, 1100])
def test_equal_calls_give_equal_bits(cuda, lib, t, N, K, T):
    """The order of an element's sum is fixed by the launch, and by the weights alone for up to 512 tokens of k-quant rows."""
    W = O.synth_blocks(t, N, K, seed=N)
    X = np.random.default_rng(K).standard_normal((T, K)).astype(np.float32)
    first = run_mmq(lib, t, W, N, K, X)
    for _ in range(3):
        assert np.array_equal(run_mmq(lib, t, W, N, K, X), first)
    if t in (O.Q4_K, O.Q5_K, O.Q6_K) and T <= 512:
        assert np.array_equal(run_mmq(lib, t, W, N, K, X[:8]), first[:8])


def test_a_prompt_in_slices_gives_the_same_bits(cuda, pkg):
    """A model wider than one cluster's tile cut, 72 tokens at once and as 40 + 32."""
    from tiny_model import TinyModel
    tm = TinyModel(n_layer=2, n_embd=2560, n_head=20, n_head_kv=4, n_ff=4096, n_vocab=256, n_ctx=96, arch="llama", ftype="q4_K_M", freq_factors=False, seed=8, branch_scale=0.1)
    toks = [(i * 31 + 7) % 256 for i in range(72)]
    out = []
    for cuts in ([72], [40, 32]):
        m, at = tm.load_engine(pkg), 0
        for n in cuts:
            got = m.prefill(toks[at:at + n], at).copy()
            at += n
        out.append(got)
        m.close()
    assert np.array_equal(out[0], out[1])
