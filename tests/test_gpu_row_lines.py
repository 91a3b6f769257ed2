"""-m gpu: prompts at the lengths from which a CTA routes eight tokens and a thread convolves four, whole groups of them and rests, against the float64 oracles."""
import numpy as np
import pytest

import ref_ludusun as RL
import ref_sapudra as RS
import ref_zevedra as RZ
import test_gpu_ludusun as L
import test_gpu_sapudra as S
import test_gpu_zevedra as Z

pytestmark = pytest.mark.gpu


def lines(lib, rows):
    """tokens up to which a token has a CTA of its own (a warp a router row, 8 to 32 of them)"""
    per_sm = 2048 // (256 if rows <= 8 else 1024 if rows >= 32 else 32 * rows)
    return lib.c.pb200_sm_count() * (per_sm if per_sm > 2 else 2 * per_sm)


@pytest.mark.parametrize("moe", [dict(experts=15, top=3, count=5, keep=2), dict(experts=32, top=4, ff=30, count=8, keep=4), dict(experts=24, top=2, ff=36, count=1, keep=1, shared=None)])
def test_routing(pkg, cuda, lib, moe):
    cfg = S.config([S.att_layer(heads=2, kv_heads=1, dim=16, vdim=16, window=40, mlp=S.moe_ff(**moe))], width=72, vocab=37, max_positions=1024)
    bits, W = RS.random_weights(cfg, seed=moe["experts"])
    m = S.load(pkg, cfg, bits, n_ctx=1024)
    line = lines(lib, moe["experts"] + (moe.get("shared", 56) is not None))
    assert line < 1000
    for n in (line, line + 1, line + 8):
        t = S.tokens_for(cfg, n, n)
        want = RS.forward(cfg, W, t)
        want = want[0] if isinstance(want, tuple) else want
        s = m.seq_alloc()
        got = m.batch_step([(s, t, list(range(n)))])[0]
        m.seq_free(s)
        assert RS.rel_err(np.asarray(got, dtype=np.float64), want).max() < S.F32_TOL, n
    m.close()


def test_convolution(pkg, cuda, lib):
    cfg = L.config([L.par(heads=2, kv_heads=1, dim=16, r_heads=8, r_kv=8, r_dim=128, r_vdim=128, taps=4, ff=0)], width=64, vocab=37)
    bits, W = RL.random_weights(cfg, seed=5)
    m = L.load(pkg, cfg, bits, n_ctx=512)
    line = -(-14 * lib.c.pb200_sm_count() // 6)      # 3072 channels: six tiles of 512
    for n in (line - 1, line, line + 1, line + 3):
        t = L.tokens_for(cfg, n, n)
        L.check(L.run_whole(m, t), RL.forward(cfg, W, t)[0], L.F32_TOL)
    m.close()


def test_more_tokens_than_a_grid_has_rows(pkg, cuda):
    """Five prompts that have more tokens together than the four-tap convolution's grid takes in groups of four, against each of them alone."""
    cfg = Z.config([Z.par(heads=1, kv_heads=1, dim=8, vdim=8, rot=4, window=16, conv=4, r_heads=1, r_kv=1, r_dim=8, r_vdim=8, r_conv=4)], width=16, vocab=23)
    bits, W = RZ.random_weights(cfg, seed=3)
    m = Z.load(pkg, cfg, bits, n_ctx=53000)
    ts = [np.random.default_rng(i).integers(0, 23, 53000).astype(np.int32) for i in range(5)]

    def run(ts):
        slots = [m.seq_alloc() for _ in ts]
        out = m.batch_step([(s, t, [20, len(t) - 1]) for s, t in zip(slots, ts)])[0].copy()
        for s in slots:
            m.seq_free(s)
        return out
    together = run(ts)
    assert np.isfinite(together).all()
    for i, t in enumerate(ts):
        assert RS.rel_err(together[2 * i:2 * i + 2].astype(np.float64), run([t]).astype(np.float64)).max() < Z.F32_TOL
    m.close()
