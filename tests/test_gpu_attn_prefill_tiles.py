"""Prompt attention over the f16 cache at the edges of the tensor-core kernel's tiles (128 positions, 128 query rows of a GQA group): group sizes that
do and do not divide 128, ragged prompts, positions in any order, cache rows that hold no numbers."""
import ctypes as C
import math

import pytest

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr())


def run(lib, q, k, v, pos, scale):
    import torch
    T, H, _ = q.shape
    out = torch.full_like(q, float("nan"))
    lib.check(lib.c.pb200_attn_prefill(ptr(q), ptr(k), ptr(v), ptr(out), H, k.shape[1], 128, ptr(pos), T, k.shape[0], scale, None), "attn_prefill")
    torch.cuda.synchronize()
    assert lib.c.pb200_aborted() == 0
    return out


def check(lib, q, k, v, pos, scale):
    """Every row against float64.  A probability rounds to f16 by 2^-11 of itself, below 2^-14 by 2^-25; its value in front of the rounding and the fp32
    sums add a fiftieth of that."""
    import torch
    out = run(lib, q, k, v, pos, scale).double()
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    see = torch.arange(k.shape[0], device="cuda")[None, :] <= pos[:, None].long()
    qh, kd, vd = q.half().double(), torch.nan_to_num(k.double(), 0, 0, 0), torch.nan_to_num(v.double(), 0, 0, 0)
    for h in range(H):
        g = h // (H // G)
        s = torch.where(see, qh[:, h] @ kd[:, g].T * scale, -math.inf)
        p = torch.nan_to_num(torch.softmax(s, -1), 0.0)
        bound = 1.02 * 2.0 ** -11 * (p @ vd[:, g].abs()) + 2.0 ** -25 * (see.double() @ vd[:, g].abs()) + 1e-7
        assert bool(((out[:, h] - p @ vd[:, g]).abs() <= bound).all()), h
    return out


def inputs(T, H, G, S, seed=0, spread=1.0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed + T * 31 + H)
    return (torch.randn(T, H, 128, generator=g, device="cuda") * spread, torch.randn(S, G, 128, generator=g, device="cuda").half(),
            torch.randn(S, G, 128, generator=g, device="cuda").half())


@pytest.mark.parametrize("H,G,T,pos0", [(4, 4, 65, 0), (4, 4, 129, 0), (8, 8, 3, 126), (6, 2, 43, 85), (6, 2, 84, 300), (8, 2, 32, 96), (8, 2, 33, 95), (64, 8, 17, 500), (20, 4, 26, 1000),
                                        (128, 1, 5, 130), (4, 1, 300, 0), (7, 1, 40, 2000)])
def test_edges_of_tiles(cuda, lib, H, G, T, pos0):
    import torch
    q, k, v = inputs(T, H, G, pos0 + T)
    check(lib, q, k, v, torch.arange(pos0, pos0 + T, dtype=torch.int32, device="cuda"), 128 ** -0.5)


def test_sharp_and_flat_scores_and_a_negative_scale(cuda, lib):
    import torch
    q, k, v = inputs(70, 8, 2, 400, spread=12.0)
    pos = torch.arange(330, 400, dtype=torch.int32, device="cuda")
    for scale in (128 ** -0.5, 0.0, -0.05):
        check(lib, q, k, v, pos, scale)


def test_positions_in_any_order(cuda, lib):
    import torch
    q, k, v = inputs(90, 8, 2, 700, seed=4)
    pos = torch.randint(0, 700, (90,), generator=torch.Generator().manual_seed(1), dtype=torch.int32).cuda()
    pos[7] = -1                       # sees nothing
    out = check(lib, q, k, v, pos, 0.1)
    assert bool((out[7] == 0).all())


def test_rows_nobody_sees_may_hold_anything(cuda, lib):
    import torch
    q, k, v = inputs(40, 8, 2, 400, seed=5)
    pos = torch.arange(100, 140, dtype=torch.int32, device="cuda")
    k[140:], v[140:] = float("nan"), float("inf")
    check(lib, q, k, v, pos, 0.1)


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
def test_a_value_that_is_no_number_stays_with_the_rows_that_see_it(cuda, lib, bad):
    import torch
    q, k, v = inputs(64, 4, 4, 264, seed=6)
    pos = torch.arange(200, 264, dtype=torch.int32, device="cuda")
    clean = run(lib, q, k, v, pos, 0.1)
    v[230, 1, 77] = bad
    out = run(lib, q, k, v, pos, 0.1)
    assert torch.equal(out[:30], clean[:30])
    assert not bool(torch.isfinite(out[30:, 1, 77]).any())
    out[30:, 1, 77] = clean[30:, 1, 77]
    assert torch.equal(out, clean)


def test_tokens_that_see_nothing(cuda, lib):
    """Whole tiles of queries before the first position: their first key tile is loaded all the same and must not reach the result."""
    import torch
    q, k, v = inputs(90, 8, 2, 300, seed=8)
    pos = torch.arange(200, 290, dtype=torch.int32, device="cuda")
    pos[32:64] = -1                   # 32 tokens x 4 heads: one CTA's rows
    for _ in range(20):
        out = check(lib, q, k, v, pos, 0.1)
        assert bool((out[32:64] == 0).all())
        assert bool((run(lib, q, k, v, torch.full_like(pos, -1), 0.1) == 0).all())


@pytest.mark.parametrize("H,G,T,pos0", [(8, 2, 21, 5), (16, 2, 6, 1790), (64, 8, 9, 120)])
@pytest.mark.parametrize("q_off,kv_off", [(1, 0), (0, 4)], ids=["queries at 4 bytes: tiled kernel", "cache at 8 bytes: one CTA per head and token"])
def test_other_alignments(cuda, lib, H, G, T, pos0, q_off, kv_off):
    import torch
    q, k, v = inputs(T, H, G, pos0 + T)

    def shifted(t, by):
        flat = torch.zeros(t.numel() + 8, dtype=t.dtype, device="cuda")
        flat[by:by + t.numel()] = t.reshape(-1)
        return flat[by:by + t.numel()].view(t.shape)
    check(lib, shifted(q, q_off), shifted(k, kv_off), shifted(v, kv_off), torch.arange(pos0, pos0 + T, dtype=torch.int32, device="cuda"), 128 ** -0.5)


def test_more_tiles_than_the_machine_holds(cuda, lib):
    """A CTA takes several items in a row: 8 tokens of 16 heads each, 51 x 8 items over at most two CTAs an SM, ragged at the end."""
    q, k, v = inputs(405, 128, 8, 405, seed=9)
    import torch
    pos = torch.arange(0, 405, dtype=torch.int32, device="cuda")
    full = check(lib, q, k, v, pos, 128 ** -0.5)
    pos[40:56] = -1                   # two items' tokens see nothing: one is its CTA's first item, one its second
    pos[392:400] = -1
    out = check(lib, q, k, v, pos, 128 ** -0.5)
    live = pos >= 0
    assert bool((out[~live] == 0).all()) and torch.equal(out[live], full[live])


def test_scores_that_grow_and_fall(cuda, lib):
    """A row's reference moves on when a tile's score is beyond it by more than 2^8: in every tile, in none behind the first, in some rows of a warp only."""
    import torch
    q, k, v = inputs(64, 8, 2, 900, seed=10)
    pos = torch.arange(836, 900, dtype=torch.int32, device="cuda")
    at = torch.arange(900, device="cuda")[:, None, None]
    for grow in (0.3 + at / 60.0, 8.0 - at / 130.0, torch.where(at // 128 % 2 == 0, 0.1, 6.0)):
        kk = (k.float() * grow).half()
        kk[:, 1] = k[:, 1]            # the second group's rows stay as they are
        check(lib, q, kk, v, pos, 128 ** -0.5)
    some = q.clone()
    some[::3] *= 0.01
    check(lib, some, (k.float() * (0.3 + at / 60.0)).half(), v, pos, 128 ** -0.5)


def test_a_score_that_is_no_number_takes_its_rows(cuda, lib):
    import torch
    q, k, v = inputs(64, 4, 4, 264, seed=11)
    pos = torch.arange(200, 264, dtype=torch.int32, device="cuda")
    clean = run(lib, q, k, v, pos, 0.1)
    for bad in (float("nan"), float("inf")):
        kb = k.clone()
        kb[230, 1] = bad              # an infinite key: products of both signs meet
        out = run(lib, q, kb, v, pos, 0.1)
        assert torch.equal(out[:30], clean[:30]) and torch.equal(out[:, [0, 2, 3]], clean[:, [0, 2, 3]])
        assert not bool(torch.isfinite(out[30:, 1]).any())
