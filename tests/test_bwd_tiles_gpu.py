"""The tensor-pipe backward with a CTA per tile, bf16 and fp32 results, at tile edges and on both sides of the lines between it and
the persistent kernels; bit-reproducible gradients have the same bits on either path (a limit on the SMs takes the persistent one)."""
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu

CASES = [
    # B, H, Sq, Sk, causal, mask, lengths, clamp
    (1, 1, 1, 1, False, False, False, 0.0),
    (2, 3, 127, 129, True, False, False, 0.0),
    (2, 2, 129, 63, True, True, True, 0.0),           # rows that see no key, a tile with none
    (3, 2, 64, 65, False, True, False, 1.0),
    (2, 2, 257, 385, True, False, True, 0.0),
    (1, 2, 128, 769, False, False, False, 0.0),       # bit-reproducible: few tiles beyond 768
    (2, 2, 640, 641, True, False, False, 1.0),
    (33, 8, 130, 100, False, False, True, 0.0),       # more tiles than fit at once
]


def _reference(q, k, v, do, causal, m, lengths, clamp):
    q, k, v, do = (t.double() for t in (q, k, v, do))
    Sq, Sk = q.shape[2], k.shape[2]
    s = q @ k.transpose(-1, -2) / 8.0
    flat = s >= clamp if clamp > 0 else torch.zeros_like(s, dtype=torch.bool)
    if clamp > 0:
        s = s.clamp(max=clamp)
    seen = torch.ones_like(s, dtype=torch.bool)
    if causal:
        seen &= torch.ones(Sq, Sk, dtype=torch.bool, device=q.device).tril(Sk - Sq)
    if m is not None:
        seen &= (m != 0)[:, None]
    if lengths is not None:
        seen &= torch.arange(Sk, device=q.device) < lengths[:, None, None, None]
    p = torch.softmax(s.masked_fill(~seen, -math.inf), -1).nan_to_num(0.0)
    dp = do @ v.transpose(-1, -2)
    ds = (p * (dp - (p * dp).sum(-1, keepdim=True)) / 8.0).masked_fill(flat, 0.0)
    return ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ do


@pytest.mark.parametrize("storage", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("case", CASES)
def test_backward_in_tiles(ctx, case, storage):
    B, H, Sq, Sk, causal, mask, lengths, clamp = case
    g = torch.Generator(device="cuda").manual_seed(9)
    rand = lambda n: (torch.randn((B, H, n, 64), generator=g, device="cuda") * 0.5).bfloat16().to(storage)   # exact bf16 values
    q, k, v, do = rand(Sq), rand(Sk), rand(Sk), rand(Sq)
    m = (torch.rand((B, Sq, Sk), generator=g, device="cuda") > 0.4).float() if mask else None
    n = torch.randint(0, Sk + 1, (B,), generator=g, device="cuda", dtype=torch.int32) if lengths else None
    if n is not None:
        n[0], n[-1] = 0, Sk
    kw = dict(causal=causal, keep_mask=m, kv_len=n, score_clamp=clamp, mode=_lib.MODE_BF16)
    o, lse = ctx.attn_fwd(q, k, v, **kw)
    want = _reference(q, k, v, do, causal, m, n, clamp)
    # the bound of the bf16 mode, half an ulp more for a result stored as bf16
    half = 2.0 ** -8 if storage == torch.bfloat16 else 0.0
    for det in (False, True):
        grads = ctx.attn_bwd(q, k, v, o, lse, do, deterministic=det, **kw)
        for name, got, ref in zip(("dq", "dk", "dv"), grads, want):
            err = (got.double() - ref).abs()
            assert bool((err <= 2e-3 * max(1.0, float(ref.abs().max())) + half * ref.abs()).all()), (name, det, float(err.max()))
    try:
        ctx.set_sm_limit(40)
        persistent = ctx.attn_bwd(q, k, v, o, lse, do, deterministic=True, **kw)
    finally:
        ctx.set_sm_limit(0)
    for a, b in zip(grads, persistent):
        assert torch.equal(a, b)
    assert ctx.device_status() == 0


# (few queries over many keys and the other way round, on both sides of the lines that keep such calls on the one-kernel form or
# the persistent pair)
@pytest.mark.parametrize("B,H,Sq,Sk,causal", [(1, 2, 100, 576, False), (1, 2, 100, 600, False), (1, 3, 128, 1024, True), (1, 2, 410, 1024, False),
                                              (1, 2, 409, 1024, False), (2, 2, 1100, 100, False), (2, 2, 1100, 800, True), (4, 8, 300, 1060, False)])
@pytest.mark.parametrize("det", [False, True])
def test_unequal_lengths(ctx, B, H, Sq, Sk, causal, det):
    g = torch.Generator(device="cuda").manual_seed(19)
    rand = lambda n: (torch.randn((B, H, n, 64), generator=g, device="cuda") * 0.5).bfloat16()
    q, k, v, do = rand(Sq), rand(Sk), rand(Sk), rand(Sq)
    o, lse = ctx.attn_fwd(q, k, v, causal=causal, mode=_lib.MODE_BF16)
    grads = ctx.attn_bwd(q, k, v, o, lse, do, causal=causal, deterministic=det, mode=_lib.MODE_BF16)
    for name, got, ref in zip(("dq", "dk", "dv"), grads, _reference(q, k, v, do, causal, None, None, 0.0)):
        err = (got.double() - ref).abs()         # as above
        assert bool((err <= 2e-3 * max(1.0, float(ref.abs().max())) + 2.0 ** -8 * ref.abs()).all()), (name, float(err.max()))
    assert ctx.device_status() == 0
