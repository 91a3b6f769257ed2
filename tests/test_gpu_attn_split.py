"""Prompt attention with every fp32 operand as two f16 numbers on the tensor cores, run inside float32 models (PB200_ATTN_SPLIT=1) where nothing else rounds
below fp32: against the float64 oracles, no further off than the fp32 FMA kernel on the same inputs, over windows, chunks, kept first tokens, soft-caps,
sinks, gates, shared key tails, another layer's cache, head sizes and groups that do not fill a tile, and lengths around the tiles of 128 positions."""
import numpy as np
import pytest

import ref_layerlist as V
import ref_ludusun as L
import ref_ruvuvik as U
import ref_zevedra as Z

pytestmark = pytest.mark.gpu


def run(pkg, monkeypatch, R, cfg, prompts, split, dtype="float32"):
    monkeypatch.setenv("PB200_ATTN_SPLIT", split)
    bits, W = R.random_weights(cfg, seed=7)
    m = pkg.Model.from_config(cfg, dtype=dtype, n_ctx=max(map(len, prompts)), n_seq=len(prompts))
    for k, b in bits.items():
        m.set_tensor(k, 30, b)
    m.finalize()
    out = m.batch_step([(m.seq_alloc(), t, list(range(len(t)))) for t in prompts])[0].astype(np.float64)
    m.close()
    return out, W


def config(arch, layers, **more):
    return dict({"architecture": arch, "width": 128, "vocab": 64, "norm": {"eps": 1e-6}, "layers": layers}, **more)


def att(H, G, D, DV=None, **more):
    return dict({"heads": H, "kv_heads": G, "dim": D, "vdim": DV or D, "scale": D ** -0.5}, **more)


def rot(dims):
    return {"base": 10000.0, "dims": dims, "scaling": {"factor": 4.0, "original": 64, "fast": 8.0, "slow": 1.0}}


def ludusun(mixer, kind="attention", times=1):
    layers = [{"type": kind, "mixer": mixer, "mlp": None}]
    if times > 1:
        layers.append({"type": kind, "mixer": dict(mixer, kv_from=0), "mlp": None})
    return L, config("Ludusun", layers, embedding={"scale": 8.0})


CASES = {
    "sink, rotation, group of 3": ludusun(att(6, 2, 64, rot=rot(64))),
    "value size 24, head size 40": ludusun(att(4, 4, 40, 24, rot=rot(40))),
    "head size 192, another layer's cache": ludusun(att(4, 2, 192, 128, rot=rot(64)), times=2),
    "latent, window 150": ludusun({"heads": 4, "dim": 128, "vdim": 100, "kv_rank": 64, "q_rank": 48, "scale": 0.1, "mask": {"size": 150}}, "latent_attention"),
    "keys are values": ludusun({"left": att(4, 1, 64), "right": att(2, 1, 32, conv=4), "left_scale": 0.7, "right_scale": 0.9}, "parallel"),
    "chunks, soft-cap": (U, config("Ruvuvik", [{"type": "attention", "mixer": att(4, 2, 32, softcap=15.0, mask={"size": 100}), "mlp": None}])),
    "shared key tail": (U, config("Ruvuvik", [{"type": "latent_attention", "mlp": None, "mixer": {"heads": 3, "dim": 100, "rot_dim": 32, "vdim": 64, "kv_rank": 64, "scale": 0.15,
                                                                                                    "rot": {"base": 10000.0, "dims": 32}}}])),
    "window 70, 5 kept tokens, gate": (V, config("Vamidra", [{"type": "attention", "mixer": att(4, 2, 128, softcap=30.0, mask={"size": 70, "keep_first": 5}), "mlp": None}], logit_scale=1.0)),
    "window 1, 140 kept tokens": (V, config("Vamidra", [{"type": "attention", "mixer": att(2, 1, 64, mask={"size": 1, "keep_first": 140}), "mlp": None}], logit_scale=1.0)),
    "sink of score 0, gate per element": (Z, config("Zevedra", [{"type": "parallel_2", "mlp": None, "mixer": {"left": att(4, 2, 64, rot={"base": 10000.0, "dims": 32}),
                                                                                                                "right": {"heads": 2, "dim": 32, "vdim": 32}}}], embedding={"scale": 8.0}, residual_mult=1.0)),
}


@pytest.mark.parametrize("name", list(CASES))
def test_no_further_from_float64_than_the_fma_kernel(pkg, cuda, monkeypatch, name):
    R, cfg = CASES[name]
    rng = np.random.default_rng(3)
    prompts = [rng.integers(0, 64, n).tolist() for n in (300, 17, 128, 1, 129, 42)]
    fma, W = run(pkg, monkeypatch, R, cfg, prompts, "0")
    split, _ = run(pkg, monkeypatch, R, cfg, prompts, "1")
    want = np.concatenate([R.forward(cfg, W, np.asarray(t))[0] for t in prompts])
    off = lambda a: np.linalg.norm(a - want) / np.linalg.norm(want)   # noqa: E731
    assert np.isfinite(split).all() and not np.array_equal(split, fma)
    # both are a few 1e-7 off; two orders of the same fp32 sums differ by a tenth of that
    assert off(split) <= 1.2 * off(fma) + 5e-8, (off(split), off(fma))
    assert np.abs(split - fma).max() < 2e-5 * np.abs(want).max()


def test_magnitudes_far_apart(pkg, cuda, monkeypatch):
    """Keys, queries and values whose rows differ by many powers of two keep their 22 bits each."""
    R, cfg = ludusun({"heads": 2, "dim": 64, "vdim": 64, "kv_rank": 64, "q_rank": 48, "scale": 1e-6, "mask": {"size": 400}}, "latent_attention")
    real = R.random_weights

    def spread(c, seed):
        bits, W = real(c, seed=seed)
        for n, lo, hi in (("uk", -12, 12), ("uv", -14, 10), ("uq", -8, 8)):
            w = W["l0.mix." + n] * 2.0 ** np.linspace(lo, hi, W["l0.mix." + n].shape[1]).round()[None, :]
            R.set_weight(bits, W, "l0.mix." + n, w)
        return bits, W
    monkeypatch.setattr(R, "random_weights", spread)
    prompts = [np.random.default_rng(4).integers(0, 64, 280).tolist()]
    fma, W = run(pkg, monkeypatch, R, cfg, prompts, "0")
    split, _ = run(pkg, monkeypatch, R, cfg, prompts, "1")
    want = R.forward(cfg, W, np.asarray(prompts[0]))[0]
    off = lambda a: np.linalg.norm(a - want) / np.linalg.norm(want)   # noqa: E731
    assert off(split) <= 1.2 * off(fma) + 5e-8, (off(split), off(fma))


def test_bfloat16_models_take_it_by_default(pkg, cuda, monkeypatch):
    R, cfg = CASES["sink, rotation, group of 3"]
    prompts = [np.random.default_rng(5).integers(0, 64, n).tolist() for n in (200, 60)]
    got, W = run(pkg, monkeypatch, R, cfg, prompts, "1", "bfloat16")
    monkeypatch.delenv("PB200_ATTN_SPLIT")
    bits, _ = R.random_weights(cfg, seed=7)
    m = pkg.Model.from_config(cfg, dtype="bfloat16", n_ctx=200, n_seq=2)
    for k, b in bits.items():
        m.set_tensor(k, 30, b)
    m.finalize()
    out = m.batch_step([(m.seq_alloc(), t, list(range(len(t)))) for t in prompts])[0]
    m.close()
    assert np.array_equal(out, got.astype(np.float32))


def loud_prompt(kind, power, tokens=128):
    """Tokens of which only the one at position 100 has something in the first width entry, which the value product (power of two, or an overflow into one
    infinite value) alone reads.  NaN: that token's embedding, hence its query, key and value, is no number."""
    R, cfg = ludusun(dict(att(4, 2, 64), scale=1.0))
    bits, W = R.random_weights(cfg, seed=11)
    emb, v = W["embed"].copy(), W["l0.mix.v"].copy()
    emb[:, 0] = 0.0
    emb[5, 0] = 8.0 * 128 ** -0.5
    v[:, 0] = 2.0 ** power * np.sign(v[:, 0]) if kind == "loud" else 0.0
    if kind == "inf":
        v[70, 0] = 3e38
    for n, w in (("embed", emb), ("l0.mix.v", v)) + tuple(("l0.mix." + n, np.where(np.arange(128) == 0, 0.0, W["l0.mix." + n])) for n in "qk"):
        R.set_weight(bits, W, n, w)
    if kind == "nan":
        bits["embed"] = bits["embed"].copy()
        bits["embed"].reshape(64, 128)[5] = 0x7fc0
    toks = np.random.default_rng(6).integers(6, 64, tokens)
    return R, cfg, bits, W, toks


def scored(pkg, cfg, bits, toks, dtype):
    m = pkg.Model.from_config(cfg, dtype=dtype, n_ctx=len(toks), n_seq=1)
    for k, b in bits.items():
        m.set_tensor(k, 30, b)
    m.finalize()
    out = m.batch_step([(m.seq_alloc(), toks.tolist(), list(range(len(toks))))])[0]
    m.close()
    return np.delete(out, 5, axis=1)   # token 5's own logit reads its embedding


@pytest.mark.parametrize("kind,power", [("loud", 12), ("loud", 24), ("loud", 40), ("loud", 100), ("inf", 0), ("nan", 0)])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_value_that_a_query_does_not_see_does_not_touch_its_row(pkg, cuda, monkeypatch, kind, power, dtype):
    monkeypatch.setenv("PB200_ATTN_SPLIT", "1")
    R, cfg, bits, W, toks = loud_prompt(kind, power)
    clean = scored(pkg, cfg, bits, toks, dtype)
    toks[100] = 5
    got = scored(pkg, cfg, bits, toks, dtype)
    assert np.array_equal(got[:100], clean[:100])
    assert not np.array_equal(got[100:], clean[100:])
    if dtype == "float32":
        want = np.delete(R.forward(cfg, W, toks[:100])[0], 5, axis=1)
        assert np.linalg.norm(got[:100] - want) <= 2e-6 * np.linalg.norm(want)
    if kind != "loud":   # one column of one kv head; the product behind it spreads it over the whole row
        assert not np.isfinite(got[100:]).any()


@pytest.mark.parametrize("power", [6, 12, 20, 28, 36])
def test_a_loud_value_of_small_weight(pkg, cuda, monkeypatch, power):
    """Scores spread over tens of binades: whatever weight the loud value has, a row is as close to float64 as with the FMA kernel, in the tile with
    rows that do not see it and behind."""
    R, cfg, bits, W, toks = loud_prompt("loud", power, 300)
    toks[100] = 5
    want = np.delete(R.forward(cfg, W, toks)[0], 5, axis=1)
    off = {}
    for split in "01":
        monkeypatch.setenv("PB200_ATTN_SPLIT", split)
        got = scored(pkg, cfg, bits, toks, "float32").astype(np.float64)
        off[split] = np.sqrt(np.mean(np.sum((got - want) ** 2, axis=1) / np.sum(want ** 2, axis=1)))
    assert off["1"] <= 1.2 * off["0"] + 5e-8, off


def test_equal_calls_give_equal_bits_whatever_ran_before(pkg, cuda, monkeypatch):
    """Many short prompts in one batch, before and after a larger batch has grown the model's work space; and the kernel that runs is the split one."""
    R, cfg = CASES["sink, rotation, group of 3"]
    rng = np.random.default_rng(8)
    short = [rng.integers(0, 64, 30).tolist() for _ in range(40)]
    bits, W = R.random_weights(cfg, seed=7)
    outs = []
    for split in ("1", "0"):
        monkeypatch.setenv("PB200_ATTN_SPLIT", split)
        m = pkg.Model.from_config(cfg, dtype="float32", n_ctx=900, n_seq=41)
        for k, b in bits.items():
            m.set_tensor(k, 30, b)
        m.finalize()
        for again in range(2):
            slots = [m.seq_alloc() for _ in short]
            outs.append(m.batch_step([(s, t, [29]) for s, t in zip(slots, short)])[0])
            for s in slots:
                m.seq_free(s)
            if not again:
                s = m.seq_alloc()
                m.batch_step([(s, rng.integers(0, 64, 900).tolist(), [0])])
                m.seq_free(s)
        m.close()
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[2], outs[3])
    assert not np.array_equal(outs[0], outs[2])


def test_more_heads_than_the_scratch_holds(pkg, cuda, monkeypatch):
    """128 key heads of 17 tiles each are 290 MB of split keys and values: they go through the scratch in two groups."""
    R, cfg = ludusun({"heads": 128, "dim": 128, "vdim": 128, "kv_rank": 32, "q_rank": 32, "scale": 0.1, "mask": {"size": 600}}, "latent_attention")
    prompts = [np.random.default_rng(9).integers(0, 64, 2100).tolist()]
    fma, _ = run(pkg, monkeypatch, R, cfg, prompts, "0")
    split, _ = run(pkg, monkeypatch, R, cfg, prompts, "1")
    assert not np.array_equal(split, fma)
    assert np.abs(split - fma).max() < 2e-5 * np.abs(fma).max()
