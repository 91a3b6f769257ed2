"""-m gpu: quantized products whose raw blocks come a K group of a row tile at a time, against the CPU oracle, where tiles, groups and the way of the
fetch change: one row, one group, more groups than the ring is deep, rows that do and do not lie at multiples of 16 bytes, a short last group."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_mmq import check, oracle, run_mmq

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t,N,K,T", [(O.Q4_K, 1, 256, 16), (O.Q4_K, 130, 1280, 17), (O.Q4_K, 257, 2048, 300), (O.Q5_K, 129, 256, 33), (O.Q5_K, 200, 1536, 520),
                                     (O.Q6_K, 129, 2048, 40), (O.Q6_K, 129, 1280, 40), (O.Q6_K, 257, 4096, 9)])
def test_groups_vs_oracle(cuda, lib, port, t, N, K, T):
    rng = np.random.default_rng(N + K + T)
    W = O.synth_blocks(t, N, K, seed=3 * t + N)
    X = rng.standard_normal((T, K)).astype(np.float32)
    check(run_mmq(lib, t, W, N, K, X), oracle(port, t, W, N, K, X), port.dequantize(t, W, N * K).reshape(N, K), X)


# Q8_0 / Q5_1 rows of 1024 and 1088 lie at multiples of 16 bytes or not, and end inside a group or not
@pytest.mark.parametrize("t,N,K,T", [(O.Q8_0, 130, 1024, 24), (O.Q8_0, 130, 1088, 24), (O.Q5_1, 130, 1088, 24), (O.Q5_1, 1, 256, 300)])
def test_small_blocks_vs_oracle(cuda, lib, port, t, N, K, T):
    rng = np.random.default_rng(N + K + T)
    W = O.synth_blocks(t, N, K, seed=3 * t + N)
    X = rng.standard_normal((T, K)).astype(np.float32)
    check(run_mmq(lib, t, W, N, K, X), oracle(port, t, W, N, K, X), port.dequantize(t, W, N * K).reshape(N, K), X)
