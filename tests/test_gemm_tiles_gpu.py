"""The tensor-pipe products' tiles at their edges, through the module that runs them: a last pair of CTAs whose second
half has no rows (6496 = 25 * 256 + 96) or lacks one (6655), columns that end inside a tile (320, 136), and products small
enough for the 128 x 128 tile."""
import math

import numpy as np
import pytest
import torch

import oracle
from cuda_ltc_b200 import _lib
from util import bf16_round, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,E,H", [(812, 8, 320, 16), (605, 11, 320, 16), (25, 8, 136, 2), (1, 3, 40, 1)])
def test_module_products(ctx, B, S, E, H):
    W, rng = 64, np.random.default_rng(B)
    HW = H * W
    lim = math.sqrt(6.0 / (E + W))
    x = bf16_round((0.5 * rng.standard_normal((B * S, E))).astype(np.float32))
    dy = bf16_round(rng.standard_normal((B * S, E)).astype(np.float32))
    w = [bf16_round(rng.uniform(-lim, lim, s).astype(np.float32)) for s in ((E, HW), (E, HW), (E, HW), (HW, E))]
    sc = 1.0 / math.sqrt(W)
    _, y_ref = oracle.tsa_fwd(x, *w, B, S, H, W, sc, True, False, False, False)
    g_ref = oracle.tsa_bwd(x, *w, dy, B, S, H, W, sc, True, False)
    d = [torch.from_numpy(a).cuda() for a in (x, *w)]
    kw = dict(scale=sc, causal=True, time_major=False, mode=_lib.MODE_BF16)
    y = ctx.tsa_fwd(*d, B, S, H, W, use_residual=False, use_layer_norm=False, **kw)
    g = ctx.tsa_bwd(*d, torch.from_numpy(dy).cuda(), B, S, H, W, **kw)
    assert ctx.device_status() == 0
    # the inputs are exact bf16 values; what is stored as bf16 between the products is off by 2^-9 of itself, at most
    # eight such results (q, k, v, P, ctx, dctx, dS, dq/dk/dv) enter one gradient
    for got, ref in zip((y, *g), (y_ref, *g_ref)):
        assert rel_l2(got.cpu().numpy(), ref) < 8 * 2.0 ** -9
