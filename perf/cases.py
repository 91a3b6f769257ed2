"""Performance cases of the framework: what its users have it do, through its public entry points, over the range of sizes in which they do
it.  Two families of models and the single operators of the C ABI:

  the k-quant family   Llama graphs over GGUF blocks (Q4_K / Q5_K / Q6_K): ``Model.prefill`` and ``Model.decode``, and the operators
                       ``pb200_mul_mat_vec`` (one token) and ``pb200_attn_prefill`` (prompt attention over the f16 cache)
  the layer lists      dense bf16 (or f32) models described by a configuration: ``Model.batch_step`` over sequence slots, as single layers
                       that score a prompt and as whole models that answer requests token by token; the operator ``pb200_dense``

A case is a dict of plain values; ``prepare`` makes what a program holds before the call (weights, inputs, slots of a model), ``run`` is one
pass, ``exact`` the same result in 64 bits from the definitions, without this package's code."""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import pkgload

DEV = "cuda"
BLOCK_BYTES = {"q4_K": 144, "q5_K": 176, "q6_K": 210}


# ---------------------------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # one attention projection of an 8B model for one token: the smallest call, the user waits for every one of them
        {"name": "gemv_q4_K_4096", "kind": "gemv", "type": "q4_K", "n": 4096, "k": 4096},
        # prompt attention of one layer of an 8B model, a 2048-token prompt from the start
        {"name": "attn_prompt_2048", "kind": "attn", "heads": 32, "kv_heads": 8, "tokens": 2048, "pos0": 0},
        # one generated token of a Q4_K_M model (four layers at 8B sizes) behind a context of a thousand tokens
        {"name": "llama_decode", "kind": "llama_decode", "layers": 4, "width": 4096, "ff": 14336, "heads": 32, "kv_heads": 8, "vocab": 32000, "mix": "q4_K", "tokens": 1000},
        # a 512-token prompt of the same model: one full batch of the prompt path
        {"name": "llama_prompt_512", "kind": "llama_prompt", "layers": 4, "width": 4096, "ff": 14336, "heads": 32, "kv_heads": 8, "vocab": 32000, "mix": "q4_K", "tokens": 512},
        # the widest product of a dense bf16 model of width 4096 (gate and up together) over a long prompt: the largest call
        {"name": "dense_prompt_2048", "kind": "dense", "t": 2048, "n": 28672, "k": 4096, "resid": False},
        # the down product of the same model for eight sequences that decode together, onto the residual stream
        {"name": "dense_batch_8", "kind": "dense", "t": 8, "n": 4096, "k": 14336, "resid": True},
        # single layers of a layer-list model of width 2048 that score a prompt: causal grouped attention with rotation and a gated feed-forward
        {"name": "layer_attention_2048", "kind": "layer", "mixer": "attention", "dtype": "bfloat16", "width": 2048, "ff": 8192, "kv_heads": 4, "dim": 128, "lens": "2048"},
        # attention over a windowed low-rank latent, three ragged prompts in one batch
        {"name": "layer_latent_ragged", "kind": "layer", "mixer": "latent", "dtype": "bfloat16", "width": 2048, "ff": 8192, "kv_heads": 16, "dim": 128, "lens": "1111,300,77"},
        # attention beside the gated delta rule, a middling prompt
        {"name": "layer_parallel_512", "kind": "layer", "mixer": "parallel", "dtype": "bfloat16", "width": 2048, "ff": 8192, "kv_heads": 4, "dim": 128, "lens": "512"},
        # windowed attention and a mixture of sixteen experts with a shared one, a batch of two prompts
        {"name": "layer_moe_ragged", "kind": "layer", "mixer": "moe", "dtype": "bfloat16", "width": 2048, "ff": 2048, "kv_heads": 4, "dim": 128, "lens": "700,324"},
        # a whole layer-list model (six layers, three mixers) answers one request: a prompt, then token by token
        {"name": "generate_b1", "kind": "generate", "width": 2048, "ff": 8192, "kv_heads": 4, "vocab": 32000, "lens": "130", "steps": 24},
        # the same model serves eight requests of different lengths together
        {"name": "generate_b8", "kind": "generate", "width": 2048, "ff": 8192, "kv_heads": 4, "vocab": 32000, "lens": "100,37,64,9,128,50,81,17", "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemv", "attn", "llama_decode", "llama_prompt", "dense", "dense", "layer", "layer", "layer", "generate"])
    if kind == "gemv":
        return {"kind": kind, "type": rng.choice(["q4_K", "q4_K", "q5_K", "q6_K"]), "n": _log_int(rng, 1000, 28672), "k": 256 * _log_int(rng, 8, 56)}
    if kind == "attn":
        kv = rng.choice([4, 8])
        tokens = _log_int(rng, 16, 2048)
        return {"kind": kind, "heads": kv * rng.choice([1, 4, 8] if kv == 4 else [1, 2, 4]), "kv_heads": kv, "tokens": tokens,
                "pos0": rng.choice([0, 0, rng.randrange(0, 2049 - tokens)])}
    if kind in ("llama_decode", "llama_prompt"):
        kv = rng.choice([2, 4, 8])
        return {"kind": kind, "layers": rng.choice([1, 2, 3]), "width": rng.choice([2048, 3072, 4096]), "ff": 256 * rng.randrange(16, 57), "heads": kv * rng.choice([2, 4]),
                "kv_heads": kv, "vocab": rng.randrange(8000, 32001), "mix": rng.choice(["q4_K", "q4_K", "q5_K"]),
                "tokens": _log_int(rng, 32, 1000) if kind == "llama_decode" else _log_int(rng, 17, 512)}
    if kind == "dense":
        big = rng.random() < 0.5
        return {"kind": kind, "t": _log_int(rng, 64, 2048) if big else rng.randrange(1, 48), "n": _log_int(rng, 700, 28672), "k": 8 * _log_int(rng, 64, 512 if big else 1792),
                "resid": rng.random() < 0.5}
    if kind == "layer":
        mixer = rng.choice(["attention", "latent", "parallel", "moe"])
        f32 = rng.random() < 0.2
        dim = rng.choice([64, 128, 128])
        heads = rng.choice([8, 12, 16] if not f32 else [4, 8])
        lens = [_log_int(rng, 20, 900 if mixer != "parallel" else 500) for _ in range(rng.choice([1, 1, 2, 3]))]
        if f32:
            lens = [min(n, 200) for n in lens[:2]]
        return {"kind": kind, "mixer": mixer, "dtype": "float32" if f32 else "bfloat16", "width": heads * dim, "ff": 8 * rng.randrange(100, 257 if f32 else 700) if mixer != "moe" else 8 * rng.randrange(50, 257),
                "kv_heads": heads // rng.choice([1, 2, 4]), "dim": dim, "lens": ",".join(str(n) for n in lens)}
    heads = rng.choice([8, 12, 16])
    lens = [_log_int(rng, 5, 130) for _ in range(rng.choice([1, 2, 4, 6, 8]))]
    return {"kind": kind, "width": 128 * heads, "ff": 8 * rng.randrange(256, 900), "kv_heads": heads // 4, "vocab": 8 * rng.randrange(500, 4001), "lens": ",".join(str(n) for n in lens),
            "steps": rng.randrange(4, 13)}


# ---------------------------------------------------------------------------------------------------------------- random inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(0x5EED + 7919 * int(seed))
    return g


def _normal(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device=DEV) * scale


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device=DEV)


def _blocks(g, type_, n, k):
    """n rows of k-quant blocks with random contents and scales that give weights of about 1 / sqrt(k): uint8 [n, k / 256, bytes]."""
    nb, sc = n * (k // 256), 1.0 / math.sqrt(k)
    raw = torch.randint(0, 256, (nb, BLOCK_BYTES[type_]), generator=g, device=DEV, dtype=torch.uint8)
    spread = _uniform(g, 0.5, 1.5, nb)
    if type_ == "q6_K":
        raw[:, 208:210] = (spread * sc / (18.0 * 64.0)).half().view(torch.uint8).view(nb, 2)
    else:
        mid = 7.5 if type_ == "q4_K" else 15.5
        d = spread * sc / (mid * 32.0)
        raw[:, 0:2] = d.half().view(torch.uint8).view(nb, 2)
        raw[:, 2:4] = (d * mid * _uniform(g, 0.9, 1.1, nb)).half().view(torch.uint8).view(nb, 2)
    return raw.view(n, k // 256, BLOCK_BYTES[type_])


def _dequantize(type_, raw):
    """uint8 [n, blocks, bytes] -> float64 [n, blocks * 256], by the definition of the block formats."""
    n, nb, _ = raw.shape
    b = raw.reshape(n * nb, -1).to(torch.int32)
    half = lambda o: raw.reshape(n * nb, -1)[:, o:o + 2].contiguous().view(torch.float16).double()   # noqa: E731  [blocks, 1]
    if type_ == "q6_K":
        ql, qh = b[:, :128].view(-1, 2, 64), b[:, 128:192].view(-1, 2, 32)
        sc = b[:, 192:208]
        sc = torch.where(sc > 127, sc - 256, sc).double().view(-1, 2, 8)
        q = torch.stack([(ql[:, :, :32] & 15) | ((qh & 3) << 4), (ql[:, :, 32:] & 15) | (((qh >> 2) & 3) << 4), (ql[:, :, :32] >> 4) | (((qh >> 4) & 3) << 4),
                         (ql[:, :, 32:] >> 4) | (((qh >> 6) & 3) << 4)], dim=2).double() - 32.0          # [blocks, 2, 4, 32]
        s = sc.view(-1, 2, 4, 2).repeat_interleave(16, dim=3)
        return (q * s * half(208).view(-1, 1, 1, 1)).reshape(n, nb * 256)
    s = b[:, 4:16]
    lo, hi, top = s[:, 0:4], s[:, 4:8], s[:, 8:12]
    scale = torch.cat([lo & 63, (top & 15) | ((lo >> 6) << 4)], dim=1).double()
    mins = torch.cat([hi & 63, (top >> 4) | ((hi >> 6) << 4)], dim=1).double()
    if type_ == "q4_K":
        qs = b[:, 16:144].view(-1, 4, 32)
        q = torch.stack([qs & 15, qs >> 4], dim=2)
    else:
        qh, qs = b[:, 16:48], b[:, 48:176].view(-1, 4, 32)
        q = torch.stack([torch.stack([(qs[:, j] & 15) + 16 * ((qh >> (2 * j)) & 1), (qs[:, j] >> 4) + 16 * ((qh >> (2 * j + 1)) & 1)], dim=1) for j in range(4)], dim=1)
    q = q.reshape(-1, 8, 32).double()
    return (q * (half(0) * scale).unsqueeze(2) - (half(2) * mins).unsqueeze(2)).reshape(n, nb * 256)


def _quantized_act(x):
    """The activation a k-quant product sees: 256 values share the scale max / -127 (q8_K), values rounded to even, float64 result."""
    b = x.float().reshape(-1, 256)
    top = b.gather(1, b.abs().argmax(dim=1, keepdim=True))
    scale = torch.where(top == 0, torch.zeros_like(top), -127.0 / top)
    q = torch.clamp(torch.round(b * scale), max=127.0)
    return torch.where(scale == 0, torch.zeros_like(q), q / scale).double().reshape(x.shape)


def _ptr(t):
    return None if t is None else C.c_void_p(t.data_ptr())


# ---------------------------------------------------------------------------------------------------------------- the k-quant family
def _llama_types(case, i):
    more = i < case["layers"] // 8 or i >= 7 * case["layers"] // 8 or (i - case["layers"] // 8) % 3 == 2   # the mixture of the _M files
    return {"attn_q": case["mix"], "attn_k": case["mix"], "attn_v": "q6_K" if more else case["mix"], "attn_output": case["mix"], "ffn_gate": case["mix"],
            "ffn_up": case["mix"], "ffn_down": "q6_K" if more else case["mix"]}


def _llama_tensors(case, seed):
    """name -> (type, rows, columns, data) of every tensor, then the tokens."""
    g = _gen(seed)
    E, F, Q, K, V = case["width"], case["ff"], 128 * case["heads"], 128 * case["kv_heads"], case["vocab"]
    shape = {"attn_q": (Q, E), "attn_k": (K, E), "attn_v": (K, E), "attn_output": (E, Q), "ffn_gate": (F, E), "ffn_up": (F, E), "ffn_down": (E, F)}
    out = {"token_embd.weight": (case["mix"], _blocks(g, case["mix"], V, E)), "output.weight": ("q6_K", _blocks(g, "q6_K", V, E)),
           "output_norm.weight": ("f32", _uniform(g, 0.9, 1.1, E))}
    for i in range(case["layers"]):
        for n, t in _llama_types(case, i).items():
            out[f"blk.{i}.{n}.weight"] = (t, _blocks(g, t, *shape[n]))
        for n in ("attn_norm", "ffn_norm"):
            out[f"blk.{i}.{n}.weight"] = ("f32", _uniform(g, 0.9, 1.1, E))
    toks = torch.randint(0, V, (case["tokens"] + 1,), generator=g, device=DEV).cpu().numpy().astype(np.int32)
    return out, toks


def _llama_exact(case, seed):
    """Logits of the last token.  Prompt and decoding see the same definition: quantized activations, keys and values kept as f16."""
    W, toks = _llama_tensors(case, seed)
    if case["kind"] == "llama_prompt":
        toks = toks[:-1]
    T, H, G, D = len(toks), case["heads"], case["kv_heads"], 128
    mul = lambda name, x: _quantized_act(x) @ _dequantize(*W[name]).T   # noqa: E731
    norm = lambda x, w: x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()   # noqa: E731
    x = _dequantize(case["mix"], W["token_embd.weight"][1][torch.as_tensor(toks, device=DEV).long()])
    ang = torch.arange(T, device=DEV).double()[:, None] * (500000.0 ** (-torch.arange(0, D, 2, device=DEV).double() / D))[None, :]
    co, si = ang.cos()[:, None, :], ang.sin()[:, None, :]

    def rope(v):
        a, b = v[..., 0::2], v[..., 1::2]
        return torch.stack([a * co - b * si, a * si + b * co], dim=-1).reshape(v.shape)
    see = torch.ones(T, T, device=DEV, dtype=torch.bool).tril()
    for i in range(case["layers"]):
        p = f"blk.{i}."
        h = norm(x, W[p + "attn_norm.weight"][1])
        q = rope(mul(p + "attn_q.weight", h).view(T, H, D)).half().double()
        k = rope(mul(p + "attn_k.weight", h).view(T, G, D)).half().double()
        v = mul(p + "attn_v.weight", h).view(T, G, D).half().double()
        o = torch.empty(T, H, D, device=DEV, dtype=torch.float64)
        for n in range(H):
            s = torch.where(see, q[:, n] @ k[:, n // (H // G)].T / math.sqrt(D), -math.inf)
            o[:, n] = torch.softmax(s, dim=-1) @ v[:, n // (H // G)]
        x = x + mul(p + "attn_output.weight", o.view(T, H * D))
        h = norm(x, W[p + "ffn_norm.weight"][1])
        x = x + mul(p + "ffn_down.weight", torch.nn.functional.silu(mul(p + "ffn_gate.weight", h)) * mul(p + "ffn_up.weight", h))
    return mul("output.weight", norm(x[-1:], W["output_norm.weight"][1]))[0]


def _prepare_llama(case, seed):
    pkg = pkgload.load()
    W, toks = _llama_tensors(case, seed)
    hp = pkg.HParams(n_layer=case["layers"], n_embd=case["width"], n_head=case["heads"], n_head_kv=case["kv_heads"], head_dim=128, n_ff=case["ff"], n_vocab=case["vocab"],
                     n_ctx=1024, rope_mode=0, n_ctx_orig=8192, rope_freq_base=500000.0, rope_freq_scale=1.0, rms_eps=1e-5)
    m = pkg.Model(hp)
    for name, (t, data) in W.items():
        m.set_tensor(name, pkg.TYPES[t], data.cpu().numpy())
    m.finalize()
    if case["kind"] == "llama_decode":
        m.prefill(toks[:-1], 0)
    return {"model": m, "tokens": toks, "logits": np.empty(case["vocab"], dtype=np.float32)}


# ---------------------------------------------------------------------------------------------------------------- the layer lists
def _mlp(ff):
    return {"kind": "dense", "ff": ff}


def _mixers(case):
    """One layer of each kind at the case's sizes, and the configuration around them."""
    H, D = case["width"] // case.get("dim", 128), case.get("dim", 128)
    G, ff = case["kv_heads"], case["ff"]
    att = {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5}
    return {
        "attention": {"type": "attention", "mlp": _mlp(ff), "mixer": dict(att, rot={"base": 1000000.0, "dims": D, "scaling": {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}})},
        "latent": {"type": "latent_attention", "mlp": _mlp(ff), "mixer": {"heads": H, "dim": D, "vdim": D, "kv_rank": 512, "q_rank": case["width"] // 2, "scale": D ** -0.5, "mask": {"size": 1024}}},
        "parallel": {"type": "parallel", "mlp": _mlp(ff),
                     "mixer": {"left": dict(att, q_temp={"coef": 0.1, "every": 512}), "right": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "conv": 4}, "left_scale": 0.7, "right_scale": 0.7}},
        "moe": {"type": "attention", "mixer": dict(att, mask={"size": 1024}),
                "mlp": {"kind": "moe", "expert": {"ff": ff}, "shared": {"ff": ff}, "router": {"experts": 16, "top": 2, "scale": 2.5, "groups": {"count": 4, "keep": 2}}}}}


def _config(case):
    mx = _mixers(case)
    if case["kind"] == "generate":   # two layers of each mixer; the second attention layer reads the first one's keys and values
        reader = dict(mx["attention"], mixer=dict(mx["attention"]["mixer"], kv_from=0))
        layers = [mx["attention"], mx["latent"], mx["parallel"], reader, mx["latent"], mx["parallel"]]
    else:
        layers = [mx[case["mixer"]]]
    cfg = {"width": case["width"], "vocab": case.get("vocab", 256), "norm": {"eps": 1e-6}, "layers": layers}
    if case.get("mixer") == "moe":
        return dict(cfg, architecture="Sapudra", max_positions=2048, residual_mult=0.5, logit_softcap=30.0)
    return dict(cfg, architecture="Ludusun", embedding={"scale": 1.0}, logit_softcap=25.0)


def _layer_tensors(cfg, g):
    """name -> float tensor (bfloat16 values) of every tensor of a configuration, with the distributions of trained layers in outline."""
    W, V, out = cfg["width"], cfg["vocab"], {}
    mat = lambda n, k: _normal(g, n, k, scale=k ** -0.5)   # noqa: E731
    moe = cfg["architecture"] == "Sapudra"
    out["embed"] = _normal(g, V, W, scale=1.0 if moe else W ** -0.5)
    if moe:
        out["pos"], out["head"], out["final.norm"], out["final.norm.b"] = _normal(g, cfg["max_positions"], W, scale=0.5), mat(V, W), 1.0 + 0.1 * _normal(g, W), 0.3 * _normal(g, W)
    else:
        out["final.norm"] = _uniform(g, -0.4, 0.4, W)
    for i, l in enumerate(cfg["layers"]):
        p, a, c = f"l{i}.", f"l{i}.mix.", l["mixer"]
        if moe:
            H, G, D, ml = c["heads"], c["kv_heads"], c["dim"], l["mlp"]
            for n in ("norm1", "norm2"):
                out[p + n], out[p + n + ".b"] = 1.0 + 0.1 * _normal(g, W), 0.3 * _normal(g, W)
            out[a + "q"], out[a + "k"], out[a + "v"], out[a + "o"] = mat(H * D, W), mat(G * D, W), mat(G * D, W), mat(W, H * D)
            out[a + "q.norm"], out[a + "k.norm"] = 1.0 + 0.1 * _normal(g, D), 1.0 + 0.1 * _normal(g, D)
            E, F = ml["router"]["experts"], ml["expert"]["ff"]
            for e in range(E):
                out[p + f"mlp.e{e}.up"], out[p + f"mlp.e{e}.down"] = mat(F, W), mat(W, F)
            out[p + "mlp.router"], out[p + "mlp.correction"] = 6.0 * mat(E, W), 0.2 * _normal(g, E)
            out[p + "mlp.shared.up"], out[p + "mlp.shared.down"], out[p + "mlp.shared.sg"] = mat(ml["shared"]["ff"], W), mat(W, ml["shared"]["ff"]), mat(1, W)
            continue
        out[p + "norm1"], out[p + "norm2"] = _uniform(g, -0.4, 0.4, W), _uniform(g, -0.4, 0.4, W)
        if l["type"] == "attention":
            H, G, D = c["heads"], c["kv_heads"], c["dim"]
            out[a + "q"], out[a + "o"], out[a + "sink"] = mat(H * D, W), mat(W, H * D), 1.5 * _normal(g, H)
            if "kv_from" not in c:
                out[a + "k"], out[a + "v"] = mat(G * D, W), mat(G * D, W)
        elif l["type"] == "latent_attention":
            H, D, R, Q = c["heads"], c["dim"], c["kv_rank"], c["q_rank"]
            out[a + "dq"], out[a + "dq.norm"], out[a + "uq"] = mat(Q, W), _uniform(g, 0.6, 1.5, Q), mat(H * D, Q)
            out[a + "dkv"], out[a + "dkv.norm"], out[a + "uk"], out[a + "uv"] = mat(R, W), _uniform(g, 0.6, 1.5, R), mat(H * D, R), mat(H * D, R)
            out[a + "g"], out[a + "o"] = mat(H, W), mat(W, H * D)
        else:
            H, G, D, lp, rp = c["left"]["heads"], c["left"]["kv_heads"], c["left"]["dim"], a + "left.", a + "right."
            out[lp + "q"], out[lp + "q.b"], out[lp + "k"], out[lp + "k.b"] = mat(H * D, W), 0.8 * _normal(g, H * D), mat(G * D, W), 0.8 * _normal(g, G * D)
            out[lp + "g"], out[lp + "o"] = mat(H * D, W), mat(W, H * D)
            for s, n in (("q", G * D), ("k", G * D), ("v", H * D)):
                out[rp + s], out[rp + s + ".conv"] = mat(n, W), 0.6 * _normal(g, n, 4)
            out[rp + "b"], out[rp + "A_log"], out[rp + "dt_bias"], out[rp + "norm"] = mat(H, W), _uniform(g, -2.0, 1.0, H), _uniform(g, -3.0, 0.5, H * D), _uniform(g, 0.6, 1.5, D)
            out[rp + "a1"], out[rp + "a2"], out[rp + "g1"], out[rp + "g2"], out[rp + "o"] = mat(D, W), mat(H * D, D), mat(D, W), mat(H * D, D), mat(W, H * D)
        out[p + "mlp.gate"], out[p + "mlp.up"], out[p + "mlp.down"] = mat(l["mlp"]["ff"], W), mat(l["mlp"]["ff"], W), mat(W, l["mlp"]["ff"])
    return {n: t.bfloat16() for n, t in out.items()}


def _layer_inputs(case, seed):
    cfg, g = _config(case), _gen(seed)
    W = _layer_tensors(cfg, g)
    lens = [int(s) for s in case["lens"].split(",")]
    toks = [torch.randint(0, cfg["vocab"], (n + case.get("steps", 0),), generator=g, device=DEV).cpu().numpy().astype(np.int32) for n in lens]
    return cfg, W, lens, toks


def _prepare_layers(case, seed):
    pkg = pkgload.load()
    cfg, W, lens, toks = _layer_inputs(case, seed)
    dtype = case.get("dtype", "bfloat16")
    m = pkg.Model.from_config(cfg, dtype=dtype, n_ctx=2048, n_seq=max(8, len(lens)))
    for name, t in W.items():
        m.set_tensor(name, pkg.TYPES["bf16"], t.view(torch.int16).cpu().numpy())
    m.finalize()
    return {"model": m, "tokens": toks, "lens": lens, "want": [np.arange(n, dtype=np.int32) for n in lens]}


def _rms(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotation(T, rot):
    dims = rot["dims"]
    i, sc = torch.arange(dims // 2, device=DEV).double(), rot["scaling"]
    f = rot["base"] ** (-2.0 * i / dims)
    place = lambda turns: dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))   # noqa: E731
    lo, hi = max(math.floor(place(sc["fast"])), 0.0), min(math.ceil(place(sc["slow"])), dims - 1.0)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    f, mag = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    a = torch.arange(T, device=DEV).double()[:, None, None] * f[None, None, :]
    return a.cos() * mag, a.sin() * mag


def _rotate(x, cs):
    half = cs[0].shape[-1]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * cs[0] - v * cs[1], v * cs[0] + u * cs[1], x[..., 2 * half:]], dim=-1)


def _attend(q, k, v, scale, window=None, sink=None):
    """q [T, H, d] over k, v [T, G, d], causal, grouped heads; sink: one more score per head in the denominator."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device=DEV)
    see = i[None, :] <= i[:, None]
    if window:
        see &= i[:, None] - i[None, :] < window
    out = torch.empty(T, H, v.shape[2], device=DEV, dtype=torch.float64)
    for h in range(H):
        s = torch.where(see, q[:, h] @ k[:, h // (H // G)].T * scale, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=-1)[:, :T] @ v[:, h // (H // G)]
    return out


def _conv(u, w):
    taps = w.shape[1]
    pad = torch.cat([torch.zeros(taps - 1, u.shape[1], device=DEV, dtype=torch.float64), u])
    return sum(pad[j:j + u.shape[0]] * w[None, :, j] for j in range(taps))


def _delta(q, k, v, g, beta):
    T, H, d = q.shape
    S, o = torch.zeros(H, d, v.shape[2], device=DEV, dtype=torch.float64), []
    for t in range(T):
        S = g[t].unsqueeze(2) * S
        u = beta[t].unsqueeze(1) * (v[t] - torch.bmm(k[t].unsqueeze(1), S).squeeze(1))
        S = torch.baddbmm(S, k[t].unsqueeze(2), u.unsqueeze(1))
        o.append(torch.bmm(q[t].unsqueeze(1), S).squeeze(1))
    return torch.stack(o)


def _ludusun_mixer(l, W, a, h, kept, i):
    T, c, sig = h.shape[0], l["mixer"], torch.sigmoid
    if l["type"] == "attention":
        H, G, D = c["heads"], c["kv_heads"], c["dim"]
        cs = _rotation(T, c["rot"])
        if "kv_from" not in c:
            kept[i] = _rms(_rotate((h @ W[a + "k"].T).view(T, G, D), cs)), (h @ W[a + "v"].T).view(T, G, D)
        k, v = kept[c.get("kv_from", i)]
        q = _rms(_rotate((h @ W[a + "q"].T).view(T, H, D), cs))
        return _attend(q, k, v, c["scale"], None, W[a + "sink"]).reshape(T, H * D) @ W[a + "o"].T
    if l["type"] == "latent_attention":
        H, D = c["heads"], c["dim"]
        cq, lat = _rms(h @ W[a + "dq"].T) * W[a + "dq.norm"], _rms(h @ W[a + "dkv"].T) * W[a + "dkv.norm"]
        o = _attend((cq @ W[a + "uq"].T).view(T, H, D), (lat @ W[a + "uk"].T).view(T, H, D), (lat @ W[a + "uv"].T).view(T, H, D), c["scale"], c["mask"]["size"])
        return (o * sig(h @ W[a + "g"].T).unsqueeze(2)).reshape(T, H * D) @ W[a + "o"].T
    lc, rc, lp, rp = c["left"], c["right"], a + "left.", a + "right."
    H, G, D = lc["heads"], lc["kv_heads"], lc["dim"]
    q, k = (h @ W[lp + "q"].T + W[lp + "q.b"]).view(T, H, D), (h @ W[lp + "k"].T + W[lp + "k.b"]).view(T, G, D)
    temp = 1.0 + lc["q_temp"]["coef"] * torch.log(torch.floor((torch.arange(T, device=DEV).double() + 1.0) / lc["q_temp"]["every"]) + 1.0)
    left = (_attend(q * temp[:, None, None], k, k, lc["scale"]).reshape(T, H * D) * sig(h @ W[lp + "g"].T)) @ W[lp + "o"].T
    q, k, v = (torch.nn.functional.silu(_conv(h @ W[rp + s].T, W[rp + s + ".conv"])) for s in "qkv")
    unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)   # noqa: E731
    q, k = (unit(q.view(T, G, D)) / math.sqrt(D)).repeat_interleave(H // G, 1), unit(k.view(T, G, D)).repeat_interleave(H // G, 1)
    dec = torch.exp(-torch.exp(W[rp + "A_log"])[None, :, None] * torch.nn.functional.softplus((h @ W[rp + "a1"].T) @ W[rp + "a2"].T + W[rp + "dt_bias"], threshold=1e9).view(T, H, D))
    o = _rms(_delta(q, k, v.view(T, H, D), dec, sig(h @ W[rp + "b"].T))) * W[rp + "norm"]
    return c["left_scale"] * left + c["right_scale"] * ((o.reshape(T, H * D) * sig((h @ W[rp + "g1"].T) @ W[rp + "g2"].T)) @ W[rp + "o"].T)


def _ludusun_exact(cfg, W, toks):
    x, kept = W["embed"][toks], {}
    for i, l in enumerate(cfg["layers"]):
        p = f"l{i}."
        x = x + _ludusun_mixer(l, W, p + "mix.", _rms(x) * (1.0 + W[p + "norm1"]), kept, i)
        h = _rms(x) * (1.0 + W[p + "norm2"])
        x = x + (torch.nn.functional.silu(h @ W[p + "mlp.gate"].T) * (h @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T
    y = (_rms(x) * (1.0 + W["final.norm"])) @ W["embed"].T
    return cfg["logit_softcap"] * torch.tanh(y / cfg["logit_softcap"])


def _sapudra_exact(cfg, W, toks):
    def ln(v, n):
        mu = v.mean(-1, keepdim=True)
        return (v - mu) / torch.sqrt(((v - mu) ** 2).mean(-1, keepdim=True) + 1e-6) * W[n] + W[n + ".b"]
    relu2 = lambda h, n: torch.relu(h @ W[n + "up"].T) ** 2 @ W[n + "down"].T   # noqa: E731
    T = len(toks)
    x = W["embed"][toks] + W["pos"][:T]
    for i, l in enumerate(cfg["layers"]):
        a, f, c, r = f"l{i}.mix.", f"l{i}.mlp.", l["mixer"], l["mlp"]["router"]
        H, G, D = c["heads"], c["kv_heads"], c["dim"]
        q, k = _rms((x @ W[a + "q"].T).view(T, H, D)) * W[a + "q.norm"], _rms((x @ W[a + "k"].T).view(T, G, D)) * W[a + "k.norm"]
        o = _attend(q, k, (x @ W[a + "v"].T).view(T, G, D), c["scale"], c["mask"]["size"])
        x = x + cfg["residual_mult"] * ln(o.reshape(T, H * D) @ W[a + "o"].T, f"l{i}.norm1")
        s = torch.sigmoid(x @ W[f + "router"].T)
        choice = (s + W[f + "correction"]).view(T, r["groups"]["count"], -1)
        best = choice.topk(2, dim=2).values.sum(2).topk(r["groups"]["keep"], dim=1).indices
        open_ = torch.zeros(T, r["groups"]["count"], device=DEV, dtype=torch.bool).scatter_(1, best, True)
        idx = torch.where(open_.unsqueeze(2), choice, -math.inf).view(T, -1).topk(r["top"], dim=1).indices
        wt = s.gather(1, idx)
        wt = wt / (wt.sum(1, keepdim=True) + 1e-20) * r["scale"]
        y = relu2(x, f + "shared.") * torch.sigmoid(x @ W[f + "shared.sg"].T)
        for e in range(r["experts"]):
            t, j = (idx == e).nonzero(as_tuple=True)
            if len(t):
                y.index_add_(0, t, wt[t, j].unsqueeze(1) * relu2(x[t], f + f"e{e}."))
        x = x + cfg["residual_mult"] * ln(y, f"l{i}.norm2")
    z = ln(x, "final.norm") @ W["head"].T
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def _layers_exact(case, seed):
    cfg, W, lens, toks = _layer_inputs(case, seed)
    W = {n: t.double() for n, t in W.items()}
    f = _sapudra_exact if cfg["architecture"] == "Sapudra" else _ludusun_exact
    logits = [f(cfg, W, torch.as_tensor(t, device=DEV).long()) for t in toks]
    if case["kind"] == "layer":
        return torch.cat(logits)
    # a step's rows: the sequences' logits after the prompt, then after every further token
    return torch.stack([torch.stack([y[n - 1 + s] for n, y in zip(lens, logits)]) for s in range(case["steps"] + 1)])


# ---------------------------------------------------------------------------------------------------------------- single operators
def _op_inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "gemv":
        return {"W": _blocks(g, case["type"], case["n"], case["k"]), "x": _normal(g, case["k"])}
    if case["kind"] == "attn":
        H, G, T, S = case["heads"], case["kv_heads"], case["tokens"], case["pos0"] + case["tokens"]
        return {"q": _normal(g, T, H, 128), "k": _normal(g, S, G, 128).half(), "v": _normal(g, S, G, 128).half()}
    T, N, K = case["t"], case["n"], case["k"]
    return {"A": _normal(g, T, K).bfloat16(), "W": _normal(g, N, K, scale=K ** -0.5).bfloat16(), "resid": _normal(g, T, N) if case["resid"] else None}


def _prepare_op(case, seed):
    lib = pkgload.load().Lib.get()
    s = dict(_op_inputs(case, seed), lib=lib, kind=case["kind"])
    if case["kind"] == "gemv":
        raw = s["W"].reshape(-1)
        s["W"] = torch.cat([raw, torch.zeros(64, dtype=torch.uint8, device=DEV)])   # the operator may read past the last row's end
        s["y"] = torch.empty(case["n"], device=DEV)
        s["ws"] = torch.zeros(lib.c.pb200_act_workspace_bytes(case["k"]) + 64, dtype=torch.uint8, device=DEV)
        s["type"] = pkgload.load().TYPES[case["type"]]
    elif case["kind"] == "attn":
        s["pos"] = torch.arange(case["pos0"], case["pos0"] + case["tokens"], dtype=torch.int32, device=DEV)
        s["y"] = torch.empty(case["tokens"], case["heads"], 128, device=DEV)
    else:
        s["y"] = torch.empty(case["t"], case["n"], device=DEV)
    s["case"] = dict(case)
    return s


def _op_exact(case, seed):
    s = _op_inputs(case, seed)
    if case["kind"] == "gemv":
        return _dequantize(case["type"], s["W"]) @ _quantized_act(s["x"])
    if case["kind"] == "attn":
        T, H, G = case["tokens"], case["heads"], case["kv_heads"]
        q, k, v = s["q"].half().double(), s["k"].double(), s["v"].double()
        see = torch.arange(case["pos0"] + T, device=DEV)[None, :] <= case["pos0"] + torch.arange(T, device=DEV)[:, None]
        out = torch.empty(T, H, 128, device=DEV, dtype=torch.float64)
        for h in range(H):
            p = torch.softmax(torch.where(see, q[:, h] @ k[:, h // (H // G)].T / math.sqrt(128), -math.inf), dim=-1)
            out[:, h] = p @ v[:, h // (H // G)]
        return out
    y = s["A"].double() @ s["W"].double().T
    return y + s["resid"].double() if s["resid"] is not None else y


# ---------------------------------------------------------------------------------------------------------------- the interface
def prepare(case, seed):
    if case["kind"] in ("llama_decode", "llama_prompt"):
        return dict(_prepare_llama(case, seed), kind=case["kind"])
    if case["kind"] in ("layer", "generate"):
        return dict(_prepare_layers(case, seed), kind=case["kind"], steps=case.get("steps", 0))
    return _prepare_op(case, seed)


def run(state):
    kind = state["kind"]
    if kind == "gemv":
        lib, c = state["lib"], state["case"]
        lib.check(lib.c.pb200_mul_mat_vec(state["type"], _ptr(state["W"]), c["n"], c["k"], _ptr(state["x"]), _ptr(state["y"]), _ptr(state["ws"]), None), "mul_mat_vec")
        return state["y"]
    if kind == "attn":
        lib, c = state["lib"], state["case"]
        lib.check(lib.c.pb200_attn_prefill(_ptr(state["q"]), _ptr(state["k"]), _ptr(state["v"]), _ptr(state["y"]), c["heads"], c["kv_heads"], 128, _ptr(state["pos"]), c["tokens"],
                                           c["pos0"] + c["tokens"], 128 ** -0.5, None), "attn_prefill")
        return state["y"]
    if kind == "dense":
        lib, c = state["lib"], state["case"]
        lib.check(lib.c.pb200_dense(30, _ptr(state["A"]), c["k"], _ptr(state["W"]), c["k"], _ptr(state["y"]), c["n"], c["t"], c["n"], c["k"], None, _ptr(state["resid"]), c["n"], 1.0,
                                    None), "dense")
        return state["y"]
    m = state["model"]
    if kind == "llama_decode":
        toks = state["tokens"]
        return m.decode(int(toks[-1]), len(toks) - 1, state["logits"])
    if kind == "llama_prompt":
        return m.prefill(state["tokens"][:-1], 0, state["logits"])
    slots = [m.seq_alloc() for _ in state["lens"]]
    try:
        if kind == "layer":
            return m.batch_step([(sl, t, w) for sl, t, w in zip(slots, state["tokens"], state["want"])])[0]
        out = [m.batch_step([(sl, t[:n], [n - 1]) for sl, t, n in zip(slots, state["tokens"], state["lens"])])[0]]
        for s in range(state["steps"]):
            out.append(m.batch_step([(sl, t[n + s:n + s + 1], [0]) for sl, t, n in zip(slots, state["tokens"], state["lens"])])[0])
        return out
    finally:
        for sl in slots:
            m.seq_free(sl)


def _layer_work(case):
    """(weight elements every token meets, weight bytes touched, attention FLOPs, recurrence FLOPs) of the layers of a case."""
    cfg, lens = _config(case), [int(s) for s in case["lens"].split(",")]
    T, W = sum(lens), cfg["width"]
    per_tok, held, other = 0, 0, 0.0
    for l in cfg["layers"]:
        c = l["mixer"]
        a = c["left"] if l["type"] == "parallel" else c
        H, D = a["heads"], a["dim"]
        G = a.get("kv_heads", H)
        win = (c.get("mask") or {}).get("size", 1 << 30)
        pairs = sum(sum(min(i + 1, win) for i in range(n + case.get("steps", 0))) for n in lens)
        other += 4.0 * H * D * pairs
        if l["type"] == "latent_attention":
            n = W * (c["q_rank"] + c["kv_rank"] + H) + H * D * (c["q_rank"] + 2 * c["kv_rank"]) + W * H * D
        elif l["type"] == "parallel":
            n = W * (2 * H * D + G * D) + W * H * D + W * (2 * G * D + H * D + H + 2 * D) + 2 * H * D * D + W * H * D
            other += 8.0 * H * D * D * (T + len(lens) * case.get("steps", 0))
        else:
            n = W * (H * D + (0 if "kv_from" in c else 2 * G * D)) + W * H * D
        if l["mlp"]["kind"] == "moe":
            f, E, top = l["mlp"]["expert"]["ff"], 16, 2
            held += n + 2 * W * f * (E + 1)
            per_tok += n + 2 * W * f * (top + 1) + W * E
        else:
            n += 3 * W * l["mlp"]["ff"]
            held += n
            per_tok += n
    return cfg, lens, per_tok, held, other


def work(case):
    kind = case["kind"]
    if kind == "gemv":
        n, k = case["n"], case["k"]
        return {"bytes": n * k // 256 * BLOCK_BYTES[case["type"]] + 4 * (n + k), "flops": 2 * n * k}
    if kind == "attn":
        T, H, G, p = case["tokens"], case["heads"], case["kv_heads"], case["pos0"]
        return {"bytes": 8 * T * H * 128 + 4 * (p + T) * G * 128, "flops": 4 * 128 * H * (T * p + T * (T + 1) // 2)}
    if kind == "dense":
        T, N, K = case["t"], case["n"], case["k"]
        return {"bytes": 2 * K * (N + T) + 4 * T * N * (2 if case["resid"] else 1), "flops": 2 * T * N * K}
    if kind in ("llama_decode", "llama_prompt"):
        E, F, Q, K, V = case["width"], case["ff"], 128 * case["heads"], 128 * case["kv_heads"], case["vocab"]
        size = {"attn_q": Q * E, "attn_k": K * E, "attn_v": K * E, "attn_output": E * Q, "ffn_gate": F * E, "ffn_up": F * E, "ffn_down": E * F}
        w = sum(size.values()) * case["layers"]
        b = sum(size[n] // 256 * BLOCK_BYTES[t] for i in range(case["layers"]) for n, t in _llama_types(case, i).items()) + V * E // 256 * BLOCK_BYTES["q6_K"] + 4 * V
        if kind == "llama_decode":
            return {"bytes": b + 4 * K * case["layers"] * (case["tokens"] + 1), "flops": 2 * (w + V * E) + 4 * Q * case["layers"] * (case["tokens"] + 1)}
        T = case["tokens"]
        return {"bytes": b + 4 * K * case["layers"] * T, "flops": 2 * w * T + 2 * V * E + 2 * Q * case["layers"] * T * (T + 1)}
    cfg, lens, per_tok, held, other = _layer_work(case)
    size = 4 if case.get("dtype") == "float32" else 2
    T, V, W = sum(lens), cfg["vocab"], cfg["width"]
    if kind == "layer":
        return {"bytes": size * (held + V * W) + 4 * T * V, "flops": 2.0 * T * (per_tok + V * W) + other}
    S = case["steps"]
    rows = len(lens) * (S + 1)
    return {"bytes": size * (held + V * W) * (S + 1) + 4 * rows * V, "flops": 2.0 * per_tok * (T + len(lens) * S) + 2.0 * rows * V * W + other}


def tolerance(case):
    """About four times what a second correct order of sums, or the 64-bit result, is away from the results of the data types in use."""
    kind = case["kind"]
    if kind == "gemv":
        return {"rel": 1e-5}                       # integer dots, sums of super-blocks in fp32
    if kind == "attn":
        return {"rel": 1e-3}                       # softmax weights rounded to f16
    if kind == "dense":
        return {"rel": 5e-5}                       # bf16 operands are exact; the tensor cores' fp32 sums over k = 14336 are 1.1e-5 off
    if kind in ("llama_decode", "llama_prompt"):
        return {"rel": 3e-2}                       # one ulp before an 8-bit activation moves it by a whole step, and all layers that follow
    if case.get("dtype") == "float32":
        return {"rel": 1e-5}
    if case.get("mixer") == "moe":
        return {"rel": 3e-2}                       # a close choice of experts may fall the other way after a rounding
    return {"rel": 2e-2 if kind == "layer" else 3e-2}


def exact(case, seed):
    if case["kind"] in ("llama_decode", "llama_prompt"):
        return _llama_exact(case, seed)
    if case["kind"] in ("layer", "generate"):
        y = _layers_exact(case, seed)
        return list(y) if case["kind"] == "generate" else y
    return _op_exact(case, seed)
