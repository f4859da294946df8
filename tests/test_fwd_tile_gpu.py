"""The tensor-pipe forward at the edges of its tiles (128 queries; 64 or 128 keys per step) and on both sides of the rule that
picks its kernel, with hidden rows, short lengths and more tiles than the GPU holds at once."""
import math

import numpy as np
import pytest
import torch

import oracle
from cuda_ltc_b200 import _lib
from util import bf16_round, max_abs, randn

pytestmark = pytest.mark.gpu

CASES = [
    # B, H, Sq, Sk, causal, lengths
    (1, 1, 1, 1, False, False),
    (2, 1, 127, 63, False, True),
    (1, 2, 128, 64, True, False),        # more queries than keys: hidden rows
    (2, 2, 129, 129, True, True),
    (1, 2, 257, 385, True, False),
    (1, 2, 300, 513, True, True),        # few tiles, long keys
    (3, 67, 260, 200, True, True),       # 603 tiles
]


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("storage", ["bf16", "f32"])
@pytest.mark.parametrize("case", CASES)
def test_forward_tiles(ctx, case, storage, D):
    B, H, Sq, Sk, causal, use_len = case
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    q, k, v = (bf16_round(randn((B, H, n, D), 50 + i, 0.5 if storage == "bf16" else 1.0)) for i, n in enumerate((Sq, Sk, Sk)))
    L = np.array([(0, Sk // 2 + 1, Sk)[i % 3] for i in range(B)], dtype=np.int32) if use_len else None
    tq, tk, tv = (torch.from_numpy(a).cuda().to(dt) for a in (q, k, v))
    o, lse = ctx.attn_fwd(tq, tk, tv, causal=causal, kv_len=torch.from_numpy(L).cuda() if use_len else None, mode=_lib.MODE_BF16)
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, 1.0 / math.sqrt(D), causal, None, L)
    # the mode's stated bound on exact bf16 inputs, half an ulp more for a result stored as bf16
    half = 2.0 ** -8 if storage == "bf16" else 0.0
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= 2e-3 + half * np.abs(o_ref)).all(), err.max()
    fin, got = np.isfinite(lse_ref), lse.cpu().numpy()
    assert (np.isfinite(got) == fin).all()
    assert max_abs(got[fin], lse_ref[fin]) < 2e-3
