"""The decode step over every way its keys are dealt out: one CTA per pair, clusters of 2 to 16 CTAs, scratch and a merge
kernel, with lengths at the edges of an iteration and of a split, and rows that start on 8-byte boundaries only."""
import math

import numpy as np
import pytest
import torch

import oracle
from util import bf16_round, max_abs, randn

pytestmark = pytest.mark.gpu

CASES = [
    # B, H, Smax, D            plan (148 SMs)
    (150, 2, 70, 64),        # one CTA of four warps per pair
    (3, 100, 513, 16),       # two CTAs of four warps
    (74, 4, 2049, 32),       # four CTAs of four warps
    (2, 3, 40, 128),         # one CTA of eight warps
    (4, 8, 129, 64),         # clusters of eight-warp CTAs
    (3, 8, 1100, 64),
    (3, 8, 4000, 128),       # sixteen
    (1, 2, 4097, 64),        # more than sixteen: scratch
]


@pytest.mark.parametrize("storage", ["f32", "bf16", "bf16_odd_rows"])
@pytest.mark.parametrize("case", CASES)
def test_decode_splits(ctx, case, storage):
    B, H, Smax, D = case
    dt = torch.float32 if storage == "f32" else torch.bfloat16
    q, k, v = (bf16_round(randn((B, H, n, D), 20 + i)) for i, n in enumerate((1, Smax, Smax)))
    edges = [0, 1, 31, 32, 33, Smax - 1, Smax, max(1, Smax // 2)]
    L = np.array([min(edges[i % len(edges)], Smax) for i in range(B)], dtype=np.int32)
    tq, tk, tv = (torch.from_numpy(a).cuda().to(dt) for a in (q, k, v))
    if storage == "bf16_odd_rows":          # row pitch D + 4: rows start on 8-byte boundaries
        tk, tv = (torch.cat([t, t[..., :4]], dim=3)[..., :D] for t in (tk, tv))
    o, lse = ctx.attn_decode(tq, tk, tv, kv_len=torch.from_numpy(L).cuda())
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, 1.0 / math.sqrt(D), False, None, L)
    # fp32 arithmetic throughout: the bound of the exact mode, half an ulp more for a result stored as bf16
    half = 0.0 if storage == "f32" else 2.0 ** -8
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= 1e-5 + half * np.abs(o_ref)).all(), err.max()
    fin = np.isfinite(lse_ref)
    got = lse.cpu().numpy()
    assert (np.isfinite(got) == fin).all()
    assert max_abs(got[fin], lse_ref[fin]) < 1e-5
