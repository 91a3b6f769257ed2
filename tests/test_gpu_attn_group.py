"""-m gpu: decode attention of the engine (a cluster of CTAs per kv head, each with a part of the cells) against numpy, at the edges of its parts:
the first cells, one chunk and one more, the buffers' end, parts of unequal length, clusters of every size."""
import ctypes as C

import numpy as np
import pytest

from tiny_model import TinyModel

pytestmark = pytest.mark.gpu
D = 128


def read(eng, lib, name, n):
    out = np.empty(n, np.float32)
    lib.check(lib.c.pb200_debug_read(eng.h, name.encode(), out.ctypes.data_as(C.c_void_p), n), "debug_read")
    return out


def rotate(x, pos, base):
    """x [..., 128], neighbouring pairs, angles by repeated fp32 multiplication; the f16 value that the cache and the scores see"""
    th, step, ang = np.float32(pos), np.float32(base ** (-2.0 / D)), np.empty(D // 2, np.float32)
    for i in range(D // 2):
        ang[i] = th
        th = np.float32(th * step)
    c, s, a, b = np.cos(ang), np.sin(ang), x[..., 0::2], x[..., 1::2]
    return np.stack([a * c - b * s, a * s + b * c], axis=-1).reshape(x.shape).astype(np.float16).astype(np.float64)


# (query heads, kv heads, n_ctx): clusters of 1, 2, 4 and 8 CTAs; groups of 2, 4 and 8 heads; 20 kv heads leave room for clusters of 4 only
@pytest.mark.parametrize("H,HK,n_ctx", [(4, 2, 64), (8, 2, 128), (16, 2, 200), (8, 4, 400), (8, 1, 1100), (4, 2, 1100), (16, 4, 1100), (40, 20, 600)])
def test_attention_of_a_step(cuda, pkg, lib, H, HK, n_ctx):
    G = H // HK
    tm = TinyModel(n_layer=1, n_embd=256, n_head=H, n_head_kv=HK, n_ff=256, n_vocab=96, n_ctx=n_ctx, seed=H + n_ctx)
    eng = tm.load_engine(pkg)
    check = {p for p in (0, 1, 7, 62, 63, 64, 65, 66, 126, 127, 128, 129, 255, 256, 300, 511, 512, 513, 519, 700, 1023, 1024, 1025, 1097, n_ctx - 1) if p < n_ctx}
    worst = 0.0
    K, V = np.empty((n_ctx, HK, D)), np.empty((n_ctx, HK, D))
    for pos in range(n_ctx):
        eng.decode((pos * 31 + 7) % 96, pos)
        K[pos] = rotate(read(eng, lib, "k", HK * D).reshape(HK, D), pos, 500000.0)
        V[pos] = read(eng, lib, "v", HK * D).reshape(HK, D).astype(np.float16)
        if pos not in check:
            continue
        q = rotate(read(eng, lib, "q", H * D).reshape(H, D), pos, 500000.0)
        got = read(eng, lib, "att", H * D).reshape(H, D)
        for h in range(H):
            s = K[:pos + 1, h // G] @ q[h] / np.sqrt(D)
            e = np.exp(s - s.max())
            p = (e / e.sum()).astype(np.float16).astype(np.float64)
            want = p @ V[:pos + 1, h // G]
            # a probability next to a rounding edge may fall the other way: 2^-11 of its term at most.  So may entries of a query or a key (their
            # angles differ in the last bits): 2^-10 of q_i k_i each, two of them in a row of scores, in the weights and in their sum
            flip = 2 * 2.0 ** -10 * np.max(np.abs(K[:pos + 1, h // G] * q[h])) / np.sqrt(D)
            assert np.all(np.abs(got[h] - want) <= (2.0 ** -11 + 2 * flip) * (p @ np.abs(V[:pos + 1, h // G])) + 1e-6), (pos, h)
            worst = max(worst, float(np.max(np.abs(got[h] - want) / (p @ np.abs(V[:pos + 1, h // G]) + 1e-6))))
    print("largest error over the sum of |terms|", worst)
    eng.close()
