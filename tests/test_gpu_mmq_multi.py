"""Products of a prompt over one activation in one launch: q, k, v and gate, up of one type and with Q6_K beside Q4_K or Q5_K, ragged rows, one and two token tiles; against
the same model token by token."""
import numpy as np
import pytest

import oracle_lib as O
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
