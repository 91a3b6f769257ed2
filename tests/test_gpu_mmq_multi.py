"""Products of a prompt over one activation in one launch: q, k, v and gate, up of one type and with Q6_K beside Q4_K or Q5_K, ragged rows, one and two token tiles; each product
against the CPU oracle, and whole prompts against the same model token by token.  Q6_K rows of 1024 entries do not lie at multiples of 16 bytes and go one by one."""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_mmq import check
from tiny_model import TinyModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ftype,types", [("q4_K_M", {}), ("q4_K_M", {"attn_v": O.Q6_K, "attn_q": O.Q4_K, "attn_k": O.Q4_K, "ffn_up": O.Q6_K}), ("q5_K_M", {"attn_q": O.Q6_K}),
                                         ("q5_K_M", {"attn_q": O.Q6_K, "attn_k": O.Q6_K, "attn_v": O.Q6_K, "ffn_gate": O.Q6_K, "ffn_up": O.Q6_K}),
                                         ("q4_K_M", {"attn_k": O.Q5_K})])   # the last one: two types, neither of them Q6_K, one after the other
@pytest.mark.parametrize("T", [9, 77, 300])
def test_prompt_against_token_by_token(cuda, pkg, ftype, types, T):
    tm = TinyModel(n_layer=2, n_embd=1024, n_head=8, n_head_kv=1, n_ff=2720 if ftype == "q5_K_M" else 2816, n_vocab=384, n_ctx=320, arch="qwen2" if ftype == "q5_K_M" else "llama",
                   ftype=ftype, types=types, seed=29, branch_scale=0.1)
    toks = [(i * 7919 + 13) % 384 for i in range(T)]
    eng = tm.load_engine(pkg)
    want = np.zeros(384, np.float32)
    for i, t in enumerate(toks):
        eng.decode(int(t), i, want)
    eng.kv_clear()
    got = [eng.prefill(toks, 0).copy() for _ in range(2)]
    eng.close()
    # as in test_gpu_engine.py: fp16 operands against integer dots
    assert float(np.sum((got[0] - want) ** 2) / np.sum(want ** 2)) < 1e-3
    assert np.array_equal(got[0], got[1])


def same(t):
    return {k: t for k in ("attn_q", "attn_k", "attn_v", "ffn_gate", "ffn_up")}


Q4, Q5, Q6 = O.Q4_K, O.Q5_K, O.Q6_K
# types, width, feed-forward rows, launches beyond the ones of both groups together: two for q, k, v one by one, one for gate and up
GROUPS = [("all_q4", same(Q4), 2048, 2816, 0), ("all_q5", same(Q5), 2048, 2752, 0), ("all_q6", same(Q6), 2048, 2752, 0),
          ("q6_beside_q4", dict(same(Q4), attn_v=Q6, ffn_up=Q6), 2048, 2752, 0), ("q6_ahead_of_q4", dict(same(Q4), attn_q=Q6, ffn_gate=Q6), 2048, 2816, 0),
          ("q6_beside_q5", dict(same(Q5), attn_k=Q6, ffn_up=Q6), 2048, 2816, 0), ("q5_between_q6", dict(same(Q6), attn_k=Q5, ffn_gate=Q5), 2048, 2752, 0),
          ("wide", dict(same(Q4), attn_v=Q6), 4096, 2816, 0),
          ("q5_beside_q4", dict(same(Q4), attn_v=Q5, ffn_up=Q5), 2048, 2816, 3), ("q6_rows_apart", dict(same(Q4), attn_v=Q6), 1024, 2816, 2)]


@pytest.mark.parametrize("name,types,E,F,apart", GROUPS, ids=[g[0] for g in GROUPS])
def test_each_product_against_the_oracle(cuda, pkg, lib, port, name, types, E, F, apart):
    H, HK = E // 128, max(1, E // 512)
    arch = "qwen2" if Q5 in types.values() else "llama"       # with biases on q, k, v
    tm = TinyModel(n_layer=1, n_embd=E, n_head=H, n_head_kv=HK, n_ff=F, n_vocab=512, n_ctx=512, arch=arch, types=types, seed=31)
    # the rotation has no angle at any position, so that what the rotating kernel leaves in q is the product; the attention's output product gives nothing, so that gate and up read
    # the normed embedding, too
    tm.tensors["rope_freqs.weight"] = (O.F32, np.full(64, 1e30, np.float32))
    tm.tensors["blk.0.attn_output.weight"] = (tm.tensors["blk.0.attn_output.weight"][0], np.zeros_like(tm.tensors["blk.0.attn_output.weight"][1]))
    eng = tm.load_engine(pkg)
    emb = port.dequantize(tm.tensors["token_embd.weight"][0], tm.tensors["token_embd.weight"][1], 512 * E).reshape(512, E).astype(np.float64)
    emb /= np.sqrt((emb * emb).mean(axis=1, keepdims=True) + tm.hp["rms_eps"])
    mats = {"q": ("attn_q", "attn_norm"), "k": ("attn_k", "attn_norm"), "v": ("attn_v", "attn_norm"), "u": ("ffn_up", "ffn_norm")}
    if F % 256 == 0:        # otherwise silu(g) * u is written over it
        mats["g"] = ("ffn_gate", "ffn_norm")
    first = {}
    for T in (512, 300, 77, 9):
        toks = [(i * 37 + 13) % 512 for i in range(T)]
        before = lib.c.pb200_kernel_launches()
        eng.prefill(toks, 0)
        # positions, embedding, q k v 2, rotation, attention, output 2, gate up 2, down 2 (and one more where its input is a kernel's of its own), head 2
        assert lib.c.pb200_kernel_launches() - before == 14 + apart + (F % 256 != 0)
        at = sorted({0, 1, 8, T // 2, T - 1} | {t for t in (63, 64, 255, 256) if t < T})
        for k, (wname, norm) in mats.items():
            t, W = tm.tensors[f"blk.0.{wname}.weight"]
            N = W.size // lib.c.pb200_row_bytes(t, E)
            got = eng.debug_read("prompt_" + k, T * N).reshape(T, N)
            assert np.array_equal(got, first.setdefault(k, got)[:T])     # a row's bits are the same with 8 and with 511 others beside it
            X = (emb[[toks[i] for i in at]] * tm.tensors[f"blk.0.{norm}.weight"][1]).astype(np.float32)
            want = np.stack([port.mul_mat(t, W, N, E, r).reshape(-1) for r in X])
            bias = tm.tensors.get(f"blk.0.{wname}.bias", (0, np.zeros(N, np.float32)))[1]
            check(got[at] - bias, want, port.dequantize(t, W, N * E).reshape(N, E), X)
    eng.close()
