"""Dense masks packed into words (attn_mask.cu) at the edges of the 32 x 32 blocks, in every tensor-pipe kernel that reads
them, and the same bits from a call whose workspace has no room for the words."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

import oracle
from cuda_ltc_b200 import _lib
from util import bf16_round, keep_mask, randn

pytestmark = pytest.mark.gpu


# (1, 2, 700, 97): several query tiles; (2, 80, 300, 161): more work items than SMs
@pytest.mark.parametrize("shape", [(2, 2, 1, 1), (1, 3, 31, 33), (2, 2, 64, 65), (1, 2, 129, 31), (1, 2, 700, 97), (2, 80, 300, 161)])
@pytest.mark.parametrize("storage", ["bf16", "f32"])
def test_masked_forward_and_backward(ctx, shape, storage):
    B, H, Sq, Sk = shape
    D = 64
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    q, k, v, do = (bf16_round(randn((B, H, n, D), 70 + i, 0.5)) for i, n in enumerate((Sq, Sk, Sk, Sq)))
    m = keep_mask(B, Sq, Sk, 3, 0.6)
    tq, tk, tv, tdo = (torch.from_numpy(a).cuda().to(dt) for a in (q, k, v, do))
    tm = torch.from_numpy(m).cuda()
    sc = 1.0 / math.sqrt(D)
    o, lse = ctx.attn_fwd(tq, tk, tv, keep_mask=tm, mode=_lib.MODE_BF16)
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, sc, False, m)
    refs = oracle.attn_bwd(q, k, v, do, sc, False, m)
    # the stated bounds of the bf16 mode (inputs are exact bf16 values), half an ulp more for a result stored as bf16
    half = 2.0 ** -8 if storage == "bf16" else 0.0
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= 2e-3 + half * np.abs(o_ref)).all(), err.max()
    fin = np.isfinite(lse_ref)
    assert (np.isfinite(lse.cpu().numpy()) == fin).all()
    for det in (False, True):
        for got, ref in zip(ctx.attn_bwd(tq, tk, tv, o, lse, tdo, keep_mask=tm, mode=_lib.MODE_BF16, deterministic=det), refs):
            err = np.abs(got.float().cpu().numpy() - ref)
            assert (err <= 2e-3 * max(1.0, np.abs(ref).max()) + half * np.abs(ref)).all(), err.max()
    if storage == "bf16":
        # no workspace at all: the kernel packs its words step by step
        o2, lse2 = torch.empty_like(o), torch.empty_like(lse)
        p = ctx._params(tq, tk, tv, o2, lse2, sc, False, tm, None, 0.0, _lib.MODE_BF16)
        ctx.check(ctx.lib.ltca_attn_fwd(ctx.handle, C.byref(p)))
        assert torch.equal(o, o2) and torch.equal(lse, lse2)
