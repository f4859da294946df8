"""The exact fp32 kernels at the sizes where their tilings can go wrong: one row beside a tile edge (32-key steps, 64- and
16-row tiles), head widths between the compiled ones, rows that are no multiple of 16 bytes, launches on both sides of the
"fills the SMs" rule, and every mask kind."""
import math

import numpy as np
import pytest
import torch

import oracle
from cuda_ltc_b200 import _lib
from util import bf16_round, keep_mask, max_abs, randn

pytestmark = pytest.mark.gpu

CASES = [
    # B, H, Sq, Sk, D, causal, mask, kvlen, clamp
    (1, 1, 1, 33, 16, False, False, False, 0.0),
    (2, 2, 31, 32, 32, True, False, False, 0.0),
    (1, 3, 65, 63, 30, False, True, True, 1.5),         # rows of 120 bytes
    (1, 2, 33, 129, 17, True, True, False, 0.0),        # element by element
    (1, 2, 64, 97, 128, True, True, True, 0.0),
    (10, 15, 65, 65, 32, True, False, False, 0.0),      # more CTAs than SMs, one row in the second tile
    (10, 15, 63, 64, 16, False, True, True, 0.5),
    (10, 15, 33, 95, 64, True, True, False, 0.0),
    (5, 30, 40, 17, 100, True, False, True, 0.0),       # more queries than keys
]


@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("case", CASES)
def test_exact_kernels_at_tile_edges(ctx, case, storage):
    B, H, Sq, Sk, D, causal, use_mask, use_len, clamp = case
    q, k, v, do = (randn((B, H, n, D), 40 + i) for i, n in enumerate((Sq, Sk, Sk, Sq)))
    dt = torch.float32
    if storage == "bf16":
        q, k, v, do = (bf16_round(a) for a in (q, k, v, do))
        dt = torch.bfloat16
    m = keep_mask(B, Sq, Sk, 5) if use_mask else None
    L = np.random.default_rng(6).integers(0, Sk + 1, size=B).astype(np.int32) if use_len else None
    sc = 1.0 / math.sqrt(D)
    dev = lambda a: torch.from_numpy(a).cuda().to(dt)
    tq, tk, tv, tdo = dev(q), dev(k), dev(v), dev(do)
    kw = dict(scale=sc, causal=causal, keep_mask=torch.from_numpy(m).cuda() if use_mask else None,
              kv_len=torch.from_numpy(L).cuda() if use_len else None, score_clamp=clamp, mode=_lib.MODE_FP32)
    o, lse = ctx.attn_fwd(tq, tk, tv, **kw)
    grads = ctx.attn_bwd(tq, tk, tv, o, lse, tdo, **kw)
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, sc, causal, m, L, clamp)
    refs = oracle.attn_bwd(q, k, v, do, sc, causal, m, L, clamp)
    # fp32 sums of at most 129 terms of magnitude about 1: 129 * 2^-24 = 8e-6.  A result stored as bf16 is off by up to
    # 2^-9 of its value, and delta = rowsum(dO o O) of the backward is formed from the rounded O: sqrt(D) * 2^-9 / sqrt(3)
    # of its terms' size, which enters dQ and dK times scale and one key's probability, below 2^-7 in all.
    half, extra = (2.0 ** -8, 2.0 ** -7) if storage == "bf16" else (0.0, 0.0)
    fin = np.isfinite(lse_ref)
    lse_h = lse.cpu().numpy().astype(np.float64)
    assert (np.isfinite(lse_h) == fin).all()
    assert max_abs(lse_h[fin], lse_ref[fin]) < 1e-5
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= 1e-5 + half * np.abs(o_ref)).all(), err.max()
    for name, got, ref in zip(("dq", "dk", "dv"), grads, refs):
        err = np.abs(got.float().cpu().numpy() - ref)
        scale = max(1.0, float(np.abs(ref).max()))
        assert (err <= (1e-5 + extra) * scale + half * np.abs(ref)).all(), (name, err.max())
    again = ctx.attn_bwd(tq, tk, tv, o, lse, tdo, **kw)
    for x, y in zip(grads, again):
        assert torch.equal(x, y)
