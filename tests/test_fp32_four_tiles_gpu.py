"""The exact backward where four 64-row tiles share an SM: more tiles than three per SM hold, narrow heads, at tile edges, both
sides of the rule's lines (mask, head width, waves, causal length, key lengths; the line that a case lies at is that of 148
SMs).  Same bounds as tests/test_fp32_tiles_gpu.py."""
import math

import numpy as np
import pytest
import torch

import oracle
from cuda_ltc_b200 import _lib
from util import keep_mask, max_abs, randn

pytestmark = pytest.mark.gpu

CASES = [
    # B, H, Sq, Sk, D, causal, mask
    (30, 15, 63, 65, 32, False, False),
    (15, 15, 65, 128, 30, True, False),
    (30, 15, 64, 64, 16, False, True),
    (30, 15, 33, 61, 9, True, True),
    (30, 15, 64, 40, 24, False, True),         # a mask and a wider head: three
    (15, 6, 257, 257, 16, True, False),        # long causal rows, too few tiles: three
    (15, 8, 250, 250, 16, True, False),        # four of them to a pair: three
    (20, 8, 180, 190, 31, True, False),        # three of them to a pair: four
    (25, 8, 250, 256, 16, True, False),        # more than five to an SM: four
    (12, 8, 399, 385, 32, False, False),       # no wave saved: three
]
LENGTH_CASES = [(25, 8, 250, 256, 16), (12, 8, 256, 250, 16), (25, 8, 250, 256, 32)]     # four; three; three


@pytest.mark.parametrize("case", CASES)
def test_exact_backward_with_many_tiles(ctx, case):
    B, H, Sq, Sk, D, causal, use_mask = case
    q, k, v, do = (randn((B, H, n, D), 50 + i) for i, n in enumerate((Sq, Sk, Sk, Sq)))
    m = keep_mask(B, Sq, Sk, 5) if use_mask else None
    sc = 1.0 / math.sqrt(D)
    dev = lambda a: torch.from_numpy(a).cuda()
    tq, tk, tv, tdo = dev(q), dev(k), dev(v), dev(do)
    kw = dict(scale=sc, causal=causal, keep_mask=dev(m) if use_mask else None, mode=_lib.MODE_FP32)
    o, lse = ctx.attn_fwd(tq, tk, tv, **kw)
    grads = ctx.attn_bwd(tq, tk, tv, o, lse, tdo, **kw)
    again = ctx.attn_bwd(tq, tk, tv, o, lse, tdo, **kw)
    refs = oracle.attn_bwd(q, k, v, do, sc, causal, m, None, 0.0)
    # fp32 sums of at most 257 terms of magnitude about 1: 257 * 2^-24 = 1.6e-5
    for name, got, rep, ref in zip(("dq", "dk", "dv"), grads, again, refs):
        assert torch.equal(got, rep), name
        assert max_abs(got.cpu().numpy(), ref) < 2e-5 * max(1.0, float(abs(ref).max())), name
    assert ctx.device_status() == 0


@pytest.mark.parametrize("case", LENGTH_CASES)
def test_exact_backward_with_many_tiles_and_key_lengths(ctx, case):
    B, H, Sq, Sk, D = case
    q, k, v, do = (randn((B, H, n, D), 55 + i) for i, n in enumerate((Sq, Sk, Sk, Sq)))
    L = np.array([(0, 1, Sk // 2, Sk)[i % 4] for i in range(B)], dtype=np.int32)
    sc = 1.0 / math.sqrt(D)
    dev = lambda a: torch.from_numpy(a).cuda()
    tq, tk, tv, tdo = dev(q), dev(k), dev(v), dev(do)
    kw = dict(scale=sc, kv_len=dev(L), mode=_lib.MODE_FP32)
    o, lse = ctx.attn_fwd(tq, tk, tv, **kw)
    grads = ctx.attn_bwd(tq, tk, tv, o, lse, tdo, **kw)
    refs = oracle.attn_bwd(q, k, v, do, sc, False, None, L, 0.0)
    for name, got, ref in zip(("dq", "dk", "dv"), grads, refs):
        assert max_abs(got.cpu().numpy(), ref) < 2e-5 * max(1.0, float(abs(ref).max())), name
    assert ctx.device_status() == 0
