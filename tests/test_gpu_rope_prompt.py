"""-m gpu: a prompt's rotation and its way into the cache in one launch against the rotation kernel and torch's conversion: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def ptr(t):
    return t.data_ptr() if t is not None else None


# (tokens, query heads, kv heads, rotated entries, mode, frequency factors): heads below, at and above the eight warps; rotated parts that end inside a half and at its edge
@pytest.mark.parametrize("T,H,HK,nd,mode,ff", [(1, 1, 1, 128, 0, False), (3, 32, 8, 128, 0, True), (5, 7, 1, 128, 2, False), (9, 40, 5, 64, 2, True), (2, 12, 3, 8, 2, False),
                                               (4, 9, 3, 8, 0, False), (6, 6, 2, 72, 0, True), (6, 6, 2, 104, 2, False)])
def test_rotation_and_store(cuda, lib, T, H, HK, nd, mode, ff):
    g = torch.Generator(device="cpu").manual_seed(nd + T)
    q, k, v = (torch.randn(T, h, 128, generator=g).cuda() for h in (H, HK, HK))
    pos = (torch.arange(T, dtype=torch.int32) * 2 + 5).cuda()
    freq = (1 + 7 * torch.rand(64, generator=g)).cuda() if ff else None
    kc, vc = (torch.full((2 * T + 8, HK, 128), 7.0, dtype=torch.float16, device="cuda") for _ in range(2))
    tail = (500000.0, 0.5, 1.0, 1.1, 32.0, 1.0, 8192, ptr(freq), None)
    wq, wk = torch.empty_like(q), torch.empty_like(k)
    lib.check(lib.c.pb200_rope(ptr(q), ptr(wq), T, H, 128, nd, mode, ptr(pos), *tail), "rope")
    lib.check(lib.c.pb200_rope(ptr(k), ptr(wk), T, HK, 128, nd, mode, ptr(pos), *tail), "rope")
    wkc, wvc = kc.clone(), vc.clone()
    wkc[pos.long()], wvc[pos.long()] = wk.half(), v.half()
    lib.check(lib.c.pb200_rope_kv_prompt(ptr(q), ptr(k), ptr(v), ptr(kc), ptr(vc), T, H, HK, nd, mode, ptr(pos), *tail), "rope_kv_prompt")
    torch.cuda.synchronize()
    assert torch.equal(q, wq) and torch.equal(kc, wkc) and torch.equal(vc, wvc)


def test_refusals(cuda, lib):
    x = torch.zeros(2, 1, 132, device="cuda")
    c = torch.zeros(8, 128, dtype=torch.float16, device="cuda")
    pos = torch.zeros(1, dtype=torch.int32, device="cuda")
    tail = (10000.0, 1.0, 0.0, 1.0, 32.0, 1.0, 4096, None, None)
    call = lambda q, nd: lib.c.pb200_rope_kv_prompt(q, ptr(x) + 528, ptr(x) + 528, ptr(c), ptr(c), 1, 1, 1, nd, 0, ptr(pos), *tail)
    assert call(ptr(x), 128) == 0
    assert call(ptr(x), 60) == -3 and call(ptr(x) + 4, 128) == -3
    assert call(None, 128) == -1 and call(ptr(x), 136) == -1
