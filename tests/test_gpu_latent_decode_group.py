"""Attention of single tokens over a latent in one kernel, against the three kernels that many sequences at once take: an odd number of heads, latents and heads that
fill their lanes and that do not, rotated parts, contexts on both sides of a cluster's and of a stage's rows; wrapped windows against the float64 oracle."""
import numpy as np
import pytest

import ref_ludusun as R
import test_gpu_ludusun as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,rot,vdim,rank", [(15, 24, 8, 28, 48), (16, 128, 0, 128, 512), (13, 100, 64, 128, 496)])
def test_one_sequence_and_many(cuda, heads, dim, rot, vdim, rank):
    import pkgload
    pkg = pkgload.load()
    mix = {"heads": heads, "dim": dim, "rot_dim": rot, "vdim": vdim, "kv_rank": rank, "q_rank": 32, "scale": (dim + rot) ** -0.5}
    if rot:
        mix["rot"] = {"base": 1e4, "dims": rot - 2}
    cfg = {"architecture": "Mumizen", "width": 128, "vocab": 96, "norm": {"eps": 1e-5, "groups": 1}, "layers": [{"type": "latent_attention", "mixer": mix, "mlp": None}]}
    m = pkg.Model.from_config(cfg, dtype="bfloat16", n_ctx=400, n_seq=16)
    m.synth(0, 11)
    m.finalize()
    toks = (np.arange(400) * 37 % 96).astype(np.int32)
    many = 97 // ((heads + 1) // 2) + 1          # more clusters than the kernel takes
    for n in (1, 7, 15, 127, 128, 129, 300):
        sl = [m.seq_alloc() for _ in range(many)]
        try:
            for s in sl:
                m.batch_step([(s, toks[:n], [n - 1])])
            want = m.batch_step([(s, toks[n:n + 1], [0]) for s in sl])[0][0].copy()
        finally:
            for s in sl:
                m.seq_free(s)
        s = m.seq_alloc()
        try:
            m.batch_step([(s, toks[:n], [n - 1])])
            got = m.batch_step([(s, toks[n:n + 1], [0])])[0][0]
        finally:
            m.seq_free(s)
        # the same fp32 numbers but for the order of sums; an entry rounded to bf16 behind them may fall the other way, by 2 ** -8 of itself
        assert np.isfinite(got).all() and np.linalg.norm(got - want) <= 2.0 ** -8 * np.linalg.norm(want)


# windows whose oldest row gives way in the middle of a CTA's share, at its ends, and a window of one row; two sequences beside each other, and then so many that the three kernels serve them
@pytest.mark.parametrize("window", [1, 16, 129, 200])
def test_wrapped_windows(pkg, cuda, window):
    cfg = L.config([L.lat(heads=5, dim=40, vdim=52, kv_rank=64, q_rank=24, window=window, ff=0), L.lat(heads=16, dim=64, vdim=64, kv_rank=512, q_rank=32, window=window, ff=264)], width=264)
    bits, W = R.random_weights(cfg, seed=window)
    m = L.load(pkg, cfg, bits, "bfloat16", n_ctx=512, n_seq=40)
    toks = L.tokens_for(cfg, 420, 5)
    want = R.forward(cfg, W, toks)[0]
    starts = [window - 1 if window > 1 else 1, 2 * window + 9]
    rows = []
    for copies in (1, 17):
        slots = [m.seq_alloc() for _ in range(2 * copies)]
        for i, s in enumerate(slots):
            m.batch_step([(s, toks[:starts[i % 2]], [])])
        got = [m.batch_step([(s, [toks[starts[i % 2] + t]], [0]) for i, s in enumerate(slots)])[0][:2].copy() for t in range(5)]
        for s in slots:
            m.seq_free(s)
        for t, g in enumerate(got):
            L.check(g, want[[n + t for n in starts]], L.BF16_TOL)
        rows.append(np.concatenate(got))
    # the same fp32 numbers but for the order of sums; of the operands rounded to bf16 behind them some fall the other way, by 2 ** -8 of an entry each, in two layers
    assert np.linalg.norm(rows[0] - rows[1]) <= 2.0 ** -7 * np.linalg.norm(rows[0])
    m.close()
