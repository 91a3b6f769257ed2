"""-m gpu: tokens whose position is advanced on the device, launched kernel by kernel without a pause between them, against the same tokens with a
synchronisation after each: a step's attention reads the position and the cells of earlier tokens ahead of its own wait.  Around the cells where the CTAs of a
cluster change their shares."""
import numpy as np
import pytest

from tiny_model import TinyModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,HK,n_ctx", [(16, 2, 300), (8, 4, 130), (4, 2, 64)])
@pytest.mark.parametrize("with_embd", [True, False])
def test_steps_in_a_row_without_graphs(cuda, pkg, H, HK, n_ctx, with_embd):
    tm = TinyModel(n_layer=2, n_embd=512, n_head=H, n_head_kv=HK, n_ff=512, n_vocab=96, n_ctx=n_ctx, seed=n_ctx)
    first = 58 if n_ctx > 70 else 50
    assert first + 12 <= n_ctx

    def run(row):
        eng = pkg.Model(pkg.HParams(**tm.hp), 0, None, with_embd, True)
        for name, (t, a) in tm.tensors.items():
            if with_embd or name != "token_embd.weight":
                eng.set_tensor(name, t, a)
        eng.finalize()
        if not with_embd:
            eng.set_hidden(np.random.default_rng(3).standard_normal(512))
        eng.set_use_graph(not row)
        eng.set_tokpos_seq(0, 7, 0)
        out = []
        for pos in range(first + 12):
            eng.step_seq_dev(0, True)
            if not row or pos in (first, first + 11):
                eng.synchronize()
            if pos in (first, first + 11):
                out.append(eng.debug_read("logits", 96))
        eng.close()
        return out
    for a, b in zip(run(True), run(False)):
        assert np.isfinite(a).all() and np.array_equal(a, b)
