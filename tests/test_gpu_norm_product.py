"""-m gpu: products of one to four bf16 tokens that make the RMS norm in front of them themselves: through models whose width does not fill a piece of a row, with biases, gated
and xIELU epilogues and gathered rows, against the float64 oracle and against the same requests in a batch of five, whose norms are kernels of their own."""
import numpy as np
import pytest

import ref_ludusun as RL
import ref_ruvuvik as RR
import test_gpu_ludusun as L
import test_gpu_ruvuvik as U

pytestmark = pytest.mark.gpu


def models(width):
    yield L, RL, L.config([L.att(heads=4, kv_heads=2, dim=64, vdim=64, rot=32, ff=300), L.lat(heads=3, dim=24, vdim=96, kv_rank=64, q_rank=32, ff=264), L.par(heads=4, r_vdim=64, ff=520)], width=width)
    yield U, RR, U.config([U.att(heads=4, kv_heads=4, dim=64, vdim=64, chunk=0, ff=264), U.lat(vdim=96, ff=296)], width=width)


@pytest.mark.parametrize("width", [256, 264, 520, 2056])
@pytest.mark.parametrize("which", [0, 1])
def test_batches_of_one_to_five(pkg, cuda, which, width):
    M, R, cfg = list(models(width))[which]
    bits, W = R.random_weights(cfg, seed=width)
    m = M.load(pkg, cfg, bits, "bfloat16", n_ctx=64)
    reqs = [M.tokens_for(cfg, 14, 30 + i) for i in range(5)]
    want = [R.forward(cfg, W, t)[0] for t in reqs]

    def steps(n):
        """prompts of one to four tokens, each alone, with wanted rows out of their middle, then steps of n requests beside each other"""
        slots, rows = [m.seq_alloc() for _ in range(n)], [[] for _ in range(n)]
        for i, s in enumerate(slots):
            k = 1 + i % 4
            rows[i] = list(m.batch_step([(s, reqs[i][:k], [k - 1] if k < 3 else [1, k - 1])])[0])
        for t in range(8):
            before = m.lib.c.pb200_kernel_launches()
            out = m.batch_step([(s, [reqs[i][1 + i % 4 + t]], [0]) for i, s in enumerate(slots)])[0]
            count = m.lib.c.pb200_kernel_launches() - before
            for i in range(n):
                rows[i].append(out[i])
        for s in slots:
            m.seq_free(s)
        return [np.stack(r) for r in rows], count

    apart, most = steps(5)
    for n in range(1, 6):
        rows, count = steps(n)
        assert count < most if n < 5 else count == most          # norms without launches of their own
        for i, got in enumerate(rows):
            k = 1 + i % 4
            at = ([k - 1] if k < 3 else [1, k - 1]) + list(range(k, k + 8))
            M.check(got, want[i][at], M.BF16_TOL)
            # fp32 numbers summed in another order; of the operands rounded to bf16 behind them, a dozen in a row, some fall the other way, by 2 ** -8 of an entry each
            assert np.linalg.norm(got - apart[i]) <= 2.0 ** -7 * np.linalg.norm(apart[i])
    m.close()


def test_more_rows_than_a_cta_keeps_sums_for(pkg, cuda):
    """A head of 152 000 rows of 256 entries: 1024 rows of two tokens' sums and 512 of four tokens' fit a CTA, which has 1028 rows."""
    cfg = L.config([L.att(heads=2, kv_heads=1, dim=32, vdim=32, ff=0)], width=256, vocab=152000)
    bits, W = RL.random_weights(cfg, seed=8)
    m = L.load(pkg, cfg, bits, "bfloat16", n_ctx=32)
    reqs = [L.tokens_for(cfg, 3, 40 + i) for i in range(5)]
    want = np.stack([RL.forward(cfg, W, t)[0][2] for t in reqs])

    def last(n):
        slots = [m.seq_alloc() for _ in range(n)]
        m.batch_step([(s, r[:2], []) for s, r in zip(slots, reqs)])
        out = m.batch_step([(s, r[2:], [0]) for s, r in zip(slots, reqs)])[0].copy()
        for s in slots:
            m.seq_free(s)
        return out
    apart = last(5)
    for n in range(1, 5):
        got = last(n)
        L.check(got, want[:n], L.BF16_TOL)
        assert np.linalg.norm(got - apart[:n]) <= 2.0 ** -7 * np.linalg.norm(apart[:n])      # as above
    m.close()


@pytest.mark.parametrize("n", [1, 3])
def test_a_profile_shows_the_kernels_that_run(pkg, cuda, n):
    cfg = list(models(520))[0][2]
    cfg["layers"] = cfg["layers"][:2]           # branches beside each other are taken one after the other while every launch is timed
    m = pkg.Model.from_config(cfg, dtype="bfloat16", n_ctx=64, n_seq=4)
    m.synth(0, 5)
    m.finalize()
    counts, rows = [], []
    for on in (False, True):
        slots = [m.seq_alloc() for _ in range(n)]
        m.batch_step([(s, [7, 9], [0]) for s in slots])
        m.profile(on)
        before = m.lib.c.pb200_kernel_launches()
        rows.append(m.batch_step([(s, [11], [0]) for s in slots])[0].copy())
        counts.append(m.lib.c.pb200_kernel_launches() - before)
        m.profile(False)
        for s in slots:
            m.seq_free(s)
    m.close()
    assert counts[0] == counts[1] and np.array_equal(rows[0], rows[1])


def test_steps_repeat(pkg, cuda):
    """The same bits however the kernels overlap: steps of one, two and four requests in turns, at a width whose pieces come from L2."""
    cfg = L.config([L.att(heads=16, kv_heads=4, dim=128, vdim=128, rot=64, ff=8192), L.lat(heads=16, dim=64, vdim=128, kv_rank=512, q_rank=256, ff=8192)], width=2048, vocab=2000)
    m = pkg.Model.from_config(cfg, dtype="bfloat16", n_ctx=64, n_seq=4)
    m.synth(0, 7)
    m.finalize()
    first = {}
    for _ in range(24):
        for n in (1, 2, 4):
            slots = [m.seq_alloc() for _ in range(n)]
            out = [m.batch_step([(s, [(31 * i + 7 * t) % 2000], [0]) for i, s in enumerate(slots)])[0].copy() for t in range(4)]
            for s in slots:
                m.seq_free(s)
            out = np.stack(out)
            assert np.isfinite(out).all() and np.array_equal(first.setdefault(n, out), out)
    m.close()
