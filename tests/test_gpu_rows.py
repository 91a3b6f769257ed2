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


# a lane has four entries of a head: full warps, part of one, heads and rotations that go to the kernels with an element a thread
@pytest.mark.parametrize("dim,vdim,rot,r_dim,r_vdim,taps", [(128, 128, 128, 128, 128, 4), (64, 32, 64, 32, 64, 4), (4, 8, 0, 4, 4, 4), (24, 20, 8, 12, 20, 3), (128, 96, 40, 100, 36, 4),
                                                            (128, 128, 4, 64, 16, 4), (132, 132, 8, 132, 132, 4), (10, 6, 2, 6, 10, 4)])
def test_heads_of_every_size(pkg, cuda, dim, vdim, rot, r_dim, r_vdim, taps):
    cfg = L.config([L.att(heads=3, kv_heads=1, dim=dim, vdim=vdim, rot=rot, ff=0), L.par(heads=4, kv_heads=2, dim=dim, r_heads=4, r_kv=2, r_dim=r_dim, r_vdim=r_vdim, taps=taps, ff=0),
                    L.att(heads=3, kv_heads=1, dim=dim, vdim=vdim, rot=rot, ff=0, of=0)], width=64, vocab=37)
    bits, W = RL.random_weights(cfg, seed=dim + taps)
    m = L.load(pkg, cfg, bits, n_ctx=256)
    for n in (1, 3, 9, 130):
        t = L.tokens_for(cfg, n, n)
        want = RL.forward(cfg, W, t)[0]
        L.check(L.run_whole(m, t), want, L.F32_TOL)
        L.check(L.run_decoded(m, t, max(1, n - 6)), want, L.F32_TOL)
    m.close()


@pytest.mark.parametrize("dtype,tol", [("float32", L.F32_TOL), ("bfloat16", L.BF16_TOL)])
@pytest.mark.parametrize("kv_rank,q_rank", [(4, 4), (64, 64), (256, 260), (512, 1024), (508, 40), (30, 20), (20, 30)])
def test_latents_of_every_size(pkg, cuda, kv_rank, q_rank, dtype, tol):
    cfg = L.config([L.lat(heads=4, dim=16, vdim=16, kv_rank=kv_rank, q_rank=q_rank, window=24, ff=0)], width=64, vocab=37)
    bits, W = RL.random_weights(cfg, seed=kv_rank)
    m = L.load(pkg, cfg, bits, dtype=dtype, n_ctx=256)
    for n in (1, 17, 45, 130):
        t = L.tokens_for(cfg, n, n)
        want = RL.forward(cfg, W, t)[0]
        L.check(L.run_whole(m, t), want, tol)
        L.check(L.run_decoded(m, t, max(1, n // 2)), want, tol)
    m.close()


@pytest.mark.parametrize("width", [72, 70])   # 70: rows that are gathered and summed an element a thread
@pytest.mark.parametrize("moe", [dict(), dict(experts=5, top=2, ff=36, count=1, keep=1, shared=None), dict(experts=32, top=4, ff=30, count=8, keep=4)])
def test_experts_of_a_prompt(pkg, cuda, width, moe):
    """Prompts of some dozens of tokens: experts with many tokens, few and none."""
    cfg = S.config([S.att_layer(heads=2, kv_heads=1, dim=16, vdim=16, window=300, mlp=S.moe_ff(**moe))], width=width, vocab=37)
    bits, W = RS.random_weights(cfg, seed=width)
    m = S.load(pkg, cfg, bits, n_ctx=256)
    for n in (63, 64, 65, 71, 72, 130):
        t = S.tokens_for(cfg, n, n)
        want = RS.forward(cfg, W, t)
        want = want[0] if isinstance(want, tuple) else want
        s = m.seq_alloc()
        got = m.batch_step([(s, t, list(range(n)))])[0]
        m.seq_free(s)
        assert RS.rel_err(np.asarray(got, dtype=np.float64), want).max() < S.F32_TOL
    m.close()
