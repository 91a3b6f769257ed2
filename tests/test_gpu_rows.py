"""-m gpu: row-wise steps with the row in registers, through small models against the float64 oracles: widths at the edges of a warp, of a row's warps
and of what the kernels take, few rows and many, and widths and head sizes that go to the kernels with an element a thread."""
import numpy as np
import pytest

import ref_ludusun as RL
import ref_sapudra as RS
import test_gpu_ludusun as L
import test_gpu_sapudra as S

pytestmark = pytest.mark.gpu

WIDTHS = [4, 36, 128, 132, 256, 516, 1020, 2052, 4100, 8192] + [30, 67, 8196]   # the last three are not taken


@pytest.mark.parametrize("width", WIDTHS)
def test_rms_norm_and_embedding(pkg, cuda, width):
    cfg = L.config([L.att(heads=2, kv_heads=1, dim=16, vdim=16, ff=24)], width=width, vocab=37)
    bits, W = RL.random_weights(cfg, seed=width)
    m = L.load(pkg, cfg, bits, n_ctx=256)
    for n in (1, 5, 127, 128, 131):
        t = L.tokens_for(cfg, n, n)
        L.check(L.run_whole(m, t), RL.forward(cfg, W, t)[0], L.F32_TOL)
    m.close()


@pytest.mark.parametrize("width", WIDTHS)
def test_layer_norm_and_residual(pkg, cuda, width):
    cfg = S.config([S.att_layer(heads=2, kv_heads=1, dim=16, vdim=16, window=300, mlp=S.dense_ff(24))], width=width, vocab=37)
    bits, W = RS.random_weights(cfg, seed=width)
    m = S.load(pkg, cfg, bits, n_ctx=256)
    for n in (1, 5, 127, 128, 131):
        t = S.tokens_for(cfg, n, n)
        want = RS.forward(cfg, W, t)
        want = want[0] if isinstance(want, tuple) else want
        s = m.seq_alloc()
        got = m.batch_step([(s, t, list(range(n)))])[0]
        m.seq_free(s)
        assert RS.rel_err(np.asarray(got, dtype=np.float64), want).max() < S.F32_TOL
    m.close()
