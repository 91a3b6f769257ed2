"""Attention of single tokens with a cluster per (entry, kv head): contexts on both sides of a cluster's and of a stage's rows, wrapped windows with kept first tokens, group sizes,
heads narrower than a warp's lanes, sinks and gates, against the prompt path of the same model, which reads no cache."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model(cuda, layer, width, n_ctx=640):
    import pkgload
    pkg = pkgload.load()
    cfg = {"architecture": "Vamidra", "width": width, "vocab": 96, "logit_scale": 1.0, "norm": {"eps": 1e-6}, "loop": {"start": 0, "stop": 1, "times": 1}, "layers": [layer]}
    m = pkg.Model.from_config(cfg, dtype="float32", n_ctx=n_ctx, n_seq=4)
    m.synth(0, 11)
    m.finalize()
    return m


@pytest.mark.parametrize("heads,kv,dim,vdim,mask,softcap", [(8, 8, 16, 16, None, 0.0), (8, 4, 64, 32, None, 30.0), (6, 2, 128, 128, {"size": 130, "keep_first": 4}, 0.0),
                                                           (8, 2, 32, 128, {"size": 200, "keep_first": 0}, 30.0), (8, 1, 128, 64, {"size": 256, "keep_first": 1}, 0.0)])
def test_steps_give_what_the_prompt_gives(cuda, heads, kv, dim, vdim, mask, softcap):
    mix = {"heads": heads, "kv_heads": kv, "dim": dim, "vdim": vdim, "scale": dim ** -0.5}
    if softcap:
        mix["softcap"] = softcap
    if mask:
        mix["mask"] = mask
    m = model(cuda, {"type": "attention", "mixer": mix, "mlp": {"kind": "dense", "ff": 64}}, 128)
    toks = (np.arange(560) * 37 % 96).astype(np.int32)
    for starts in ((1, 8), (31, 255), (256, 297), (513, 129)):   # two sequences beside each other, six steps each
        sl = [m.seq_alloc() for _ in starts]
        try:
            for s, n in zip(sl, starts):
                m.batch_step([(s, toks[:n], [n - 1])])
            got = [m.batch_step([(s, toks[n + i:n + i + 1], [0]) for s, n in zip(sl, starts)])[0].copy() for i in range(6)]
        finally:
            for s in sl:
                m.seq_free(s)
        for k, n in enumerate(starts):
            s = m.seq_alloc()
            try:
                want = m.batch_step([(s, toks[:n + 6], np.arange(n, n + 6))])[0]
            finally:
                m.seq_free(s)
            have = np.stack([g[k] for g in got])
            # fp32 throughout, sums of up to 560 terms in another order: 560 / 2 ** 24 = 3e-5 a side in the mixer, and as much again in the products behind it
            assert np.linalg.norm(have - want) <= 1e-4 * np.linalg.norm(want)
