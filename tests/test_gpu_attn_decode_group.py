"""Attention of single tokens with a cluster per (entry, kv head): contexts on both sides of a cluster's and of a stage's rows, wrapped windows with kept first tokens, group sizes,
heads narrower than a warp's lanes, against the prompt path of the same model, which reads no cache; sinks, chunks that are crossed, keys that are their own values over more rows than
the stages of a cluster hold, and bf16, against the float64 oracles."""
import numpy as np
import pytest

import ref_ludusun as RL
import ref_ruvuvik as RR
import test_gpu_ludusun as L
import test_gpu_ruvuvik as U

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


# a cluster holds 1024 rows of keys that are their own values, 512 of keys and values: starts on both sides; chunks of 130 and 200 whose ends are crossed
CASES = {"tied": (L, RL, lambda: L.config([L.par(heads=4, kv_heads=2, dim=64, every=300, ff=0)]), (1021, 1085, 127)),
         "tied_one_head": (L, RL, lambda: L.config([L.par(heads=3, kv_heads=3, dim=128, every=0, ff=0)]), (1024, 1281)),
         "sinks": (L, RL, lambda: L.config([L.att(heads=8, kv_heads=1, dim=96, vdim=64, ff=0)]), (508, 545, 31)),
         "sinks_read_by_another_layer": (L, RL, lambda: L.config([L.att(heads=4, kv_heads=2, dim=32, vdim=128, ff=0), L.att(heads=8, kv_heads=2, dim=32, vdim=128, of=0, scale=0.7, ff=24)]), (255, 513)),
         "chunks": (U, RR, lambda: U.config([U.att(heads=4, kv_heads=2, dim=64, vdim=64, chunk=130, rot=0, ff=0)]), (127, 257, 387)),
         "chunks_of_200": (U, RR, lambda: U.config([U.att(heads=6, kv_heads=6, dim=32, vdim=40, chunk=200, ff=0)]), (196, 200, 397))}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_steps_give_what_the_oracle_gives(pkg, cuda, name, dtype):
    M, R, cfg, starts = CASES[name]
    cfg = cfg()
    bits, W = R.random_weights(cfg, seed=17)
    m = M.load(pkg, cfg, bits, dtype, n_ctx=1300)
    toks = M.tokens_for(cfg, max(starts) + 6, 3)
    want = R.forward(cfg, W, toks)[0]
    slots = [m.seq_alloc() for _ in starts]
    for s, n in zip(slots, starts):
        m.batch_step([(s, toks[:n], [n - 1])])
    for i in range(6):
        got = m.batch_step([(s, [toks[n + i]], [0]) for s, n in zip(slots, starts)])[0]
        M.check(got, want[[n + i for n in starts]], M.F32_TOL if dtype == "float32" else M.BF16_TOL)
    m.close()
