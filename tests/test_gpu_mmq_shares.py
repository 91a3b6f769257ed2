"""-m gpu: the k-quant product where a CTA's share of the work begins and ends in each of the ways its rule allows.

Bound: the element-wise fp16-roundings bound and NMSE of test_gpu_mmq.check; a split adds one fp32 rounding per CTA of the tile, far below it.
"""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_mmq import check, oracle, run_mmq

pytestmark = pytest.mark.gpu


# (rows, K, tokens): on 148 SMs a share of one group of several, two tiles, a share that ends inside tiles, one whole tile, and the edges of
# the 16-token chunks that the 16 reading warps take (1, 15, 17 tokens; a second accumulator with one token; rows that end inside a tile)
@pytest.mark.parametrize("N,K,T", [(200, 2048, 1), (130, 3072, 15), (128, 4096, 17), (20480, 512, 17), (3840, 2816, 257), (14336, 256, 31), (129, 1024, 513)])
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
