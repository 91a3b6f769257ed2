"""-m gpu: the delta rule of single tokens against the float64 oracle: every head size, tiles of columns that are not full, two sequences beside each other, decays that are
nothing."""
import numpy as np
import pytest

import ref_ludusun as R
from test_gpu_ludusun import F32_TOL, check, config, load, par, tokens_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vdim", [(32, 8), (64, 20), (128, 32), (128, 68), (256, 36)])
@pytest.mark.parametrize("nothing", [False, True])
def test_token_by_token(pkg, cuda, dim, vdim, nothing):
    cfg = config([par(r_heads=4, r_kv=2, r_dim=dim, r_vdim=vdim, ff=0)], width=32, vocab=31)
    bits, W = R.random_weights(cfg, seed=43)
    if nothing:
        R.set_weight(bits, W, "l0.mix.right.A_log", np.full_like(W["l0.mix.right.A_log"], 6.0))
    m = load(pkg, cfg, bits, n_seq=4)
    reqs = [tokens_for(cfg, 9, 1), tokens_for(cfg, 12, 2)]
    slots = [m.seq_alloc() for _ in reqs]
    rows = [[], []]
    for i in range(12):     # the shorter one ends first
        live = [k for k in range(2) if i < len(reqs[k])]
        out = m.batch_step([(slots[k], [reqs[k][i]], [0]) for k in live])[0]
        for j, k in enumerate(live):
            rows[k].append(out[j].copy())
    for k in range(2):
        check(np.stack(rows[k]), R.forward(cfg, W, reqs[k])[0], F32_TOL)
    m.close()
