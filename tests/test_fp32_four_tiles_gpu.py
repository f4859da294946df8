"""The exact backward with many tiles of narrow heads, at tile edges: by one pass over the scores, and by the two kernels, which calls
without room for dQ's shares take (with and without room for the mask's words).  Same bounds as tests/test_fp32_tiles_gpu.py."""
import ctypes as C
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
    (30, 15, 64, 40, 24, False, True),
    (15, 6, 257, 257, 16, True, False),
    (15, 8, 250, 250, 16, True, False),
    (20, 8, 180, 190, 31, True, False),
    (25, 8, 250, 256, 16, True, False),
    (12, 8, 399, 385, 32, False, False),
]
LENGTH_CASES = [(25, 8, 250, 256, 16), (12, 8, 256, 250, 16), (25, 8, 250, 256, 32)]
# the two kernels: a workspace of delta alone or of delta and the mask's words; storage
TWO_KERNEL_CASES = [
    # B, H, Sq, Sk, D, causal, mask, words, storage
    (15, 15, 65, 129, 30, True, True, False, torch.float32),
    (15, 15, 65, 129, 30, True, True, True, torch.float32),
    (20, 8, 180, 190, 16, False, True, True, torch.float32),
    (20, 8, 180, 190, 16, True, False, False, torch.bfloat16),
    (10, 16, 127, 193, 64, True, False, False, torch.float32),
    (10, 16, 127, 193, 64, False, True, True, torch.bfloat16),
    (4, 1, 3000, 70, 32, False, False, True, torch.float32),       # many queries, few keys: too few CTAs for one pass
    (4, 1, 3000, 70, 50, True, True, True, torch.float32),
]


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


@pytest.mark.parametrize("case", TWO_KERNEL_CASES)
def test_two_kernel_backward(ctx, case):
    B, H, Sq, Sk, D, causal, use_mask, words, dt = case
    q, k, v, do = (torch.from_numpy(randn((B, H, n, D), 60 + i)).cuda().to(dt) for i, n in enumerate((Sq, Sk, Sk, Sq)))
    m = keep_mask(B, Sq, Sk, 5) if use_mask else None
    tm = torch.from_numpy(m).cuda() if use_mask else None
    sc = 1.0 / math.sqrt(D)
    o, lse = ctx.attn_fwd(q, k, v, scale=sc, causal=causal, keep_mask=tm, mode=_lib.MODE_FP32)
    p = ctx._params(q, k, v, o, lse, sc, causal, tm, None, 0.0, _lib.MODE_FP32)
    align = lambda n: (n + 255) // 256 * 256
    nbytes = align(4 * B * H * Sq)
    if words:
        room = align(4 * B * (Sq * ((Sk + 31) // 32) + Sk * ((Sq + 31) // 32)))          # by query and by key
        one = (Sk + 63) // 64 * Sq * ((D + 3) // 4 * 4) * 4
        assert 3 * (room // one) * ((Sk + 63) // 64) < 148                               # not enough for shares of dQ
        nbytes += room
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    grads = [torch.empty_like(t) for t in (q, k, v)]
    p.workspace, p.workspace_bytes = ws.data_ptr(), nbytes
    p.dout, p.do_strides = do.data_ptr(), _lib.Strides(*do.stride()[:3])
    for name, t in zip(("dq", "dk", "dv"), grads):
        setattr(p, name, t.data_ptr())
        setattr(p, name + "_strides", _lib.Strides(*t.stride()[:3]))
    ctx.check(ctx.lib.ltca_attn_bwd(ctx.handle, C.byref(p)))
    host = lambda t: t.float().cpu().numpy()
    refs = oracle.attn_bwd(host(q), host(k), host(v), host(do), sc, causal, m, None, 0.0)
    for name, got, ref in zip(("dq", "dk", "dv"), grads, refs):
        # fp32 sums of up to 3000 terms: 3000 * 2^-24 at most, the few hundred of the other cases 2e-5; bf16 results are rounded once,
        # and delta comes from a bf16 output
        mag = max(1.0, float(abs(ref).max()))
        tol = 2e-4 if max(Sq, Sk) > 1000 else 2e-5
        assert max_abs(host(got), ref) < (tol + (2.0 ** -7 if dt == torch.bfloat16 else 0.0)) * mag, name
    assert ctx.device_status() == 0
