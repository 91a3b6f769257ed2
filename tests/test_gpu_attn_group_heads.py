"""-m gpu: decode attention of the engine at the edges of its two layouts (a head a CTA for short contexts, the cells over a cluster for longer ones) and of the
chunks the short one loads; heads of several kv heads in one cluster.  Queries and keys are rotated by the library, so that they are the kernel's own."""
import ctypes as C

import numpy as np
import pytest
import torch

from gpu_util import dev_f32, ptr, sync
from test_gpu_attn_group import D, read
from tiny_model import TinyModel

pytestmark = pytest.mark.gpu
EDGES = (0, 1, 15, 16, 62, 63, 64, 65, 126, 127, 128, 129, 190, 191, 192, 193, 254, 255, 256, 257, 258, 320, 521)


def rotated(lib, x, heads, pos, mode):
    """[heads, 128] as the cache and the scores see it"""
    xd, p = dev_f32(x), torch.tensor([pos], dtype=torch.int32, device="cuda")
    y = torch.empty_like(xd)
    lib.check(lib.c.pb200_rope(ptr(xd), ptr(y), 1, heads, D, D, mode, ptr(p), 500000.0 if mode == 0 else 1000000.0, 1.0, 0.0, 1.0, 32.0, 1.0, 8192, None, None), "rope")
    sync()
    return y.cpu().numpy().reshape(heads, D).astype(np.float16).astype(np.float64)


# (query heads, kv heads, n_ctx): groups of 2, 4 and 8; clusters of 2, 4 and 8 CTAs, as many as a group has heads and more; 12 heads leave a cluster of
# eight half idle
@pytest.mark.parametrize("H,HK,n_ctx,arch", [(8, 4, 258, "llama"), (16, 8, 526, "qwen2"), (12, 6, 526, "llama"), (8, 2, 300, "qwen2"), (24, 6, 526, "llama"), (16, 2, 526, "llama"),
                                             (40, 20, 300, "llama")])
def test_edges_of_the_layouts(cuda, pkg, lib, H, HK, n_ctx, arch):
    G = H // HK
    tm = TinyModel(n_layer=1, n_embd=256, n_head=H, n_head_kv=HK, n_ff=256, n_vocab=96, n_ctx=n_ctx, seed=H + n_ctx, arch=arch)
    eng = tm.load_engine(pkg)
    K, V = np.empty((n_ctx, HK, D)), np.empty((n_ctx, HK, D))
    for pos in range(n_ctx):
        eng.decode((pos * 31 + 7) % 96, pos)
        K[pos] = rotated(lib, read(eng, lib, "k", HK * D), HK, pos, tm.hp["rope_mode"])
        V[pos] = read(eng, lib, "v", HK * D).reshape(HK, D).astype(np.float16)
        if pos not in EDGES and pos != n_ctx - 1:
            continue
        q = rotated(lib, read(eng, lib, "q", H * D), H, pos, tm.hp["rope_mode"])
        got = read(eng, lib, "att", H * D).reshape(H, D)
        for h in range(H):
            k, v = K[:pos + 1, h // G], V[:pos + 1, h // G]
            s = k @ q[h] / np.sqrt(D)
            e = np.exp(s - s.max())
            p = (e / e.sum()).astype(np.float16).astype(np.float64)
            # every probability may fall to the other side of its rounding edge: a step of f16, 2^-10 of it or 2^-24; sums of 32 bits beside that
            bound = (2.0 ** -10 + 2.0 ** -18) * (p @ np.abs(v)) + 2.0 ** -24 * np.abs(v).sum(axis=0) + 1e-7
            assert np.all(np.abs(got[h] - p @ v) <= bound), (pos, h, float(np.max(np.abs(got[h] - p @ v) / bound)))
    eng.close()
