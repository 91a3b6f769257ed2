"""Prompt attention on split operands over prompts long enough for the ring of key and value pieces to go round many times, for every number of 64-wide
units that a head has: against the fp32 FMA kernel, at the bound of the short prompts' test, and with the first rows the same bits whatever follows."""
import numpy as np
import pytest

from test_gpu_attn_split import V, att, config, ludusun, rot, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,vdim,window", [(64, 64, 0), (64, 128, 0), (128, 128, 0), (128, 64, 333), (192, 128, 0), (192, 64, 500), (100, 72, 129)])
def test_long_prompts(pkg, cuda, monkeypatch, dim, vdim, window):
    R, cfg = ludusun(att(4, 2, dim, vdim, rot=rot(32)))
    if window:
        R, cfg = V, config("Vamidra", [{"type": "attention", "mixer": att(4, 2, dim, vdim, mask={"size": window, "keep_first": 3}), "mlp": None}], logit_scale=1.0)
    rng = np.random.default_rng(dim + vdim)
    prompts = [rng.integers(0, 64, n).tolist() for n in (1153, 511, 640)]
    fma, _ = run(pkg, monkeypatch, R, cfg, prompts, "0")
    split, _ = run(pkg, monkeypatch, R, cfg, prompts, "1")
    assert np.isfinite(split).all() and not np.array_equal(split, fma)
    assert np.abs(split - fma).max() < 2e-5 * np.abs(fma).max()    # as for the short prompts: both are fp32 sums in two orders
    short, _ = run(pkg, monkeypatch, R, cfg, [prompts[0][:700]], "1")
    assert np.array_equal(short, split[:700])
