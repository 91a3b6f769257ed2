"""-m gpu: the delta rule in blocks of four tokens (prompts of a few entries) against the float64 oracle: decays that are nothing, close to one and
far apart within a head, rests of blocks and chunks, tiles of columns that are not full, and batches on both sides of the hand-over."""
import numpy as np
import pytest

import ref_ludusun as R
from test_gpu_ludusun import F32_TOL, check, config, load, par, run_whole, silenced, tokens_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vdim", [(32, 8), (64, 20), (128, 16), (256, 36)])
@pytest.mark.parametrize("decay", ["nothing", "one", "apart"])
def test_decays_of_every_size(pkg, cuda, dim, vdim, decay):
    cfg = config([par(r_heads=2, r_kv=1, r_dim=dim, r_vdim=vdim, ff=0)], width=32, vocab=31)
    bits, W = R.random_weights(cfg, seed=41)
    silenced(bits, W, cfg, 0, "left")
    a = "l0.mix.right."
    if decay == "nothing":      # exp(-exp(6) softplus): zero from the second token on
        R.set_weight(bits, W, a + "A_log", np.full_like(W[a + "A_log"], 6.0))
    elif decay == "one":
        R.set_weight(bits, W, a + "A_log", np.full_like(W[a + "A_log"], -9.0))
    else:                       # neighbouring channels forget at once and hardly at all
        R.set_weight(bits, W, a + "dt_bias", np.where(np.arange(W[a + "dt_bias"].size) % 3 == 0, 30.0, -20.0).reshape(W[a + "dt_bias"].shape))
    m = load(pkg, cfg, bits, n_seq=4)
    for n in (3, 4, 5, 7, 15, 16, 17, 19, 20, 33, 50):
        t = tokens_for(cfg, n, n)
        check(run_whole(m, t), R.forward(cfg, W, t)[0], F32_TOL)
    m.close()


def test_both_sides_of_the_hand_over(pkg, cuda):
    # 12 heads x 2 tiles of columns: one entry goes in blocks, twelve are more CTAs than SMs and go token by token; both continue token by token
    cfg = config([par(r_heads=12, r_kv=4, r_dim=32, r_vdim=24, ff=0)], width=32, vocab=31)
    bits, W = R.random_weights(cfg, seed=42)
    m = load(pkg, cfg, bits, n_seq=12)
    reqs = [tokens_for(cfg, 21 + i, i) for i in range(12)]
    slots = [m.seq_alloc() for _ in reqs]
    many = m.batch_step([(s, r, list(range(len(r)))) for s, r in zip(slots, reqs)])[0]
    at = 0
    for s, r in zip(slots, reqs):
        want = R.forward(cfg, W, r + [5, 6])[0]
        check(many[at:at + len(r)], want[:len(r)], F32_TOL)
        at += len(r)
        rest = [m.batch_step([(s, [t], [0])])[0] for t in (5, 6)]
        m.seq_free(s)
        check(np.concatenate([run_whole(m, r)] + rest), want, F32_TOL)
    m.close()
