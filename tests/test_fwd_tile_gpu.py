"""The tensor-pipe forward at the edges of its tiles (128 queries; 64 or 128 keys per step) and on both sides of the rule that
picks its kernel, with hidden rows, short lengths and more tiles than the GPU holds at once."""
import math

import numpy as np
import pytest
import torch

import oracle
from cuda_ltc_b200 import _lib
from util import bf16_round, keep_mask, max_abs, randn

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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("storage", ["bf16", "f32"])
@pytest.mark.parametrize("causal", [False, True])
def test_forward_tiles_that_rescale_at_every_step(ctx, causal, storage, D):
    """Scores that grow along the keys, by more than the 2^8 a row's running maximum may lag behind in every step of 64 or
    128 keys, so that each step rescales what it has summed up."""
    B, H, S = 2, 24, 1000
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    q, k, v = (randn((B, H, S, D), 70 + i, 0.5) for i in range(3))
    q[..., 0], k[..., 0] = 1.0, 0.125 * np.arange(S)           # natural units: 8 in 64 keys, log(2^8) = 5.5
    q, k, v = (bf16_round(a) for a in (q, k, v))
    tq, tk, tv = (torch.from_numpy(a).cuda().to(dt) for a in (q, k, v))
    o, lse = ctx.attn_fwd(tq, tk, tv, scale=1.0, causal=causal, mode=_lib.MODE_BF16)
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, 1.0, causal)
    # Exact bf16 inputs.  Results stored as bf16: probabilities and results rounded once each to 8 significant bits, which is
    # 2^-8 of sum P |v| and of the result.  fp32: two terms of the probabilities, 2^-16.  Both: scores up to 200 in fp32, whose rounding reaches the exponent as
    # 200 x 2^-23 at most, and the exponential's own error, together below 1e-4 of sum P |v|.
    mag = oracle.attn_fwd(q, k, np.abs(v), 1.0, causal)[0]
    bound = (2.0 ** -8 + 1e-4) * mag + 2.0 ** -8 * np.abs(o_ref) if storage == "bf16" else (2.0 ** -16 + 1e-4) * mag
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= bound + 1e-6).all(), (err.max(), (err / (bound + 1e-6)).max())
    assert max_abs(lse.cpu().numpy(), lse_ref) < 1e-3
    for _ in range(20):
        again = ctx.attn_fwd(tq, tk, tv, scale=1.0, causal=causal, mode=_lib.MODE_BF16)
        assert torch.equal(o, again[0]) and torch.equal(lse, again[1])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("storage", ["bf16", "f32"])
@pytest.mark.parametrize("case", [(1, 1, 1, 1, False, False), (2, 3, 129, 65, False, False), (2, 2, 128, 256, True, False),
                                  (2, 2, 257, 130, True, True), (3, 67, 200, 200, False, False), (2, 3, 300, 1000, False, False)])
def test_forward_tiles_with_a_mask(ctx, case, storage, D):
    """A dense mask with a hidden row, short lengths and, from 1000 keys on, scores that grow by more than 2^8 in every step, so
    that each step rescales what it has summed up."""
    B, H, Sq, Sk, causal, use_len = case
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    q, k, v = (randn((B, H, n, D), 80 + i, 0.5) for i, n in enumerate((Sq, Sk, Sk)))
    if Sk >= 1000:
        q[..., 0], k[..., 0] = 1.0, 0.125 * np.arange(Sk)
    q, k, v = (bf16_round(a) for a in (q, k, v))
    m = keep_mask(B, Sq, Sk, 7)
    L = np.array([(Sk // 2 + 1, Sk)[i % 2] for i in range(B)], dtype=np.int32) if use_len else None
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()
    tq, tk, tv = (dev(a).to(dt) for a in (q, k, v))
    o, lse = ctx.attn_fwd(tq, tk, tv, scale=0.5, causal=causal, keep_mask=dev(m), kv_len=dev(L), mode=_lib.MODE_BF16)
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, 0.5, causal, m, L)
    # as in the test above: exact bf16 inputs, probabilities in one term or two, scores up to 100
    mag = oracle.attn_fwd(q, k, np.abs(v), 0.5, causal, m, L)[0]
    bound = (2.0 ** -8 + 1e-4) * mag + 2.0 ** -8 * np.abs(o_ref) if storage == "bf16" else (2.0 ** -16 + 1e-4) * mag
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= bound + 1e-6).all(), (err.max(), (err / (bound + 1e-6)).max())
    fin, got = np.isfinite(lse_ref), lse.cpu().numpy()
    assert not fin[0, :, 0].any() and (np.isfinite(got) == fin).all()
    assert max_abs(got[fin], lse_ref[fin]) < 1e-3
    assert ctx.device_status() == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("storage", ["bf16", "f32"])
def test_forward_tiles_in_groups_of_pairs(ctx, storage, D):
    """K and V of 99 (batch, head) pairs, 50 MB in bf16, are dealt out in two groups, the last one smaller."""
    B, H, Sq, Sk = 3, 33, 260, 131072 // D
    dt = torch.bfloat16 if storage == "bf16" else torch.float32
    q, k, v = (bf16_round(randn((B, H, n, D), 90 + i, 0.5)) for i, n in enumerate((Sq, Sk, Sk)))
    tq, tk, tv = (torch.from_numpy(a).cuda().to(dt) for a in (q, k, v))
    o, lse = ctx.attn_fwd(tq, tk, tv, causal=True, mode=_lib.MODE_BF16)
    o_ref, lse_ref = oracle.attn_fwd(q, k, v, 1.0 / math.sqrt(D), True)
    half = 2.0 ** -8 if storage == "bf16" else 0.0
    err = np.abs(o.float().cpu().numpy() - o_ref)
    assert (err <= 2e-3 + half * np.abs(o_ref)).all(), err.max()
    assert max_abs(lse.cpu().numpy(), lse_ref) < 2e-3


LIMIT_CASES = [
    # B, H, Sq, Sk, causal, lengths, mask
    (1, 1, 1, 1, False, False, False),          # fewer tiles than one CTA has teams
    (3, 67, 260, 200, True, True, False),       # 603 tiles, some without keys, odd numbers of key steps
    (2, 40, 515, 515, True, False, True),
]


@pytest.mark.parametrize("n_sms", [1, 100])
@pytest.mark.parametrize("case", LIMIT_CASES)
def test_forward_under_an_sm_limit_has_the_same_bits(ctx, case, n_sms):
    B, H, Sq, Sk, causal, use_len, use_mask = case
    q, k, v = (torch.from_numpy(randn((B, H, n, 64), 60 + i, 0.5)).cuda().bfloat16() for i, n in enumerate((Sq, Sk, Sk)))
    kw = dict(causal=causal, mode=_lib.MODE_BF16)
    if use_len:
        kw["kv_len"] = torch.tensor([(0, Sk // 2 + 1, Sk)[i % 3] for i in range(B)], dtype=torch.int32, device="cuda")
    if use_mask:
        kw.update(keep_mask=(torch.rand((B, Sq, Sk), device="cuda") > 0.2).float(), score_clamp=1.0)
    want = ctx.attn_fwd(q, k, v, **kw)
    try:
        ctx.set_sm_limit(n_sms)
        got = [ctx.attn_fwd(q, k, v, **kw) for _ in range(2)]      # (twice: the tile counter is back at zero)
    finally:
        ctx.set_sm_limit(0)
    torch.cuda.synchronize()
    assert ctx.device_status() == 0
    for o, lse in got:
        assert torch.equal(o, want[0]) and torch.equal(lse, want[1])


def test_forward_keeps_to_the_sm_limit(ctx):
    """On an eighteenth of the SMs a call that fills the GPU many times over takes far longer."""
    q, k, v = ((torch.randn((4, 40, 1024, 64), device="cuda") * 0.5).bfloat16() for _ in range(3))

    def best():
        times = []
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            ctx.attn_fwd(q, k, v, mode=_lib.MODE_BF16)
            b.record()
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    free = best()
    try:
        ctx.set_sm_limit(8)
        held = best()
    finally:
        ctx.set_sm_limit(0)
    assert held > 4 * free, (held, free)
