"""Attention of single tokens over a latent in one kernel, against the three kernels that many sequences at once take: an odd number of heads, latents and heads that
fill their lanes and that do not, rotated parts, contexts on both sides of a cluster's and of a stage's rows."""
import numpy as np
import pytest

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
