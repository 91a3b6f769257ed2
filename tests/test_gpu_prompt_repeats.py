"""-m gpu: a prompt gives the same bits however its kernels overlap: layers at the sizes of an 8B model, the prompt again and again, with prompts of other lengths between."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
E = 4096


def hidden(m, n):
    class View:
        __cuda_array_interface__ = {"shape": (n, E), "typestr": "<i4", "data": (m.lib.c.pb200_prefill_hidden_device(m.h), False), "version": 2}
    return torch.as_tensor(View(), device="cuda").clone()


@pytest.mark.parametrize("ftype", [0, 1])          # Q4_K and Q5_K with Q6_K among them
def test_prompts_repeat(cuda, pkg, ftype):
    hp = pkg.HParams(n_layer=3, n_embd=E, n_head=32, n_head_kv=8, head_dim=128, n_ff=14336, n_vocab=1024, n_ctx=1024, rope_mode=0, n_ctx_orig=8192, rope_freq_base=500000.0,
                     rope_freq_scale=1.0, rms_eps=1e-5)
    m = pkg.Model(hp)
    m.synth(ftype, 7)
    m.finalize()
    first, differ = {}, {}
    for i in range(24):
        for n in (512, 100, 88, 250, 17, 40):
            m.prefill((np.arange(n) * 31 + 7) % 1024, 0)
            x = hidden(m, n)
            if n not in first:
                first[n] = x
            elif not torch.equal(first[n], x):
                differ[n] = differ.get(n, 0) + 1
    m.close()
    assert not differ, differ
