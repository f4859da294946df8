"""The one-pass exact backward: key blocks of 64 with a remainder, one block or several, query tiles that no key of a block sees,
every mask, strided operands that no vector load takes, and more (batch, head) pairs than one launch has room for.  Against
PyTorch in 64 bits."""
import ctypes as C
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu

CASES = [
    # B, H, Sq, Sk, D, causal, mask, lengths, clamp, storage
    (40, 4, 64, 64, 32, False, False, False, 0.0, torch.float32),      # one block: dQ is written where it belongs
    (40, 4, 70, 33, 16, True, False, False, 0.0, torch.float32),       # one block, rows that see no key
    (40, 4, 5, 61, 9, False, True, True, 0.0, torch.float32),
    (20, 4, 65, 129, 32, True, False, False, 0.0, torch.float32),      # a last block of one key
    (20, 4, 200, 100, 30, True, True, False, 1.0, torch.float32),      # more queries than keys; no vector loads
    (10, 8, 130, 250, 64, False, True, True, 1.0, torch.float32),
    (8, 8, 191, 193, 64, True, False, True, 0.0, torch.float32),
    (10, 8, 127, 128, 18, False, True, False, 0.0, torch.bfloat16),
]


def _reference(q, k, v, do, scale, causal, m, lengths, clamp):
    """dq, dk, dv and the largest sum of magnitudes behind an element of each."""
    q, k, v, do = (t.double() for t in (q, k, v, do))
    Sq, Sk = q.shape[2], k.shape[2]
    s = q @ k.transpose(-1, -2) * scale
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
    ds = (p * (dp - (p * dp).sum(-1, keepdim=True)) * scale).masked_fill(flat, 0.0)
    grads = ds @ k, ds.transpose(-1, -2) @ q, p.transpose(-1, -2) @ do
    mags = ds.abs() @ k.abs(), ds.abs().transpose(-1, -2) @ q.abs(), p.transpose(-1, -2) @ do.abs()
    return grads, [float(x.max()) for x in mags]


@pytest.mark.parametrize("case", CASES)
def test_one_pass_backward(ctx, case):
    B, H, Sq, Sk, D, causal, mask, lengths, clamp, dt = case
    g = torch.Generator(device="cuda").manual_seed(5)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda").to(dt)
    q, k, v, do = rand(B, H, Sq, D), rand(B, H, Sk, D), rand(B, H, Sk, D), rand(B, H, Sq, D)
    m = (torch.rand((B, Sq, Sk), generator=g, device="cuda") > 0.4).float() if mask else None
    n = torch.randint(0, Sk + 1, (B,), generator=g, device="cuda", dtype=torch.int32) if lengths else None
    if n is not None:
        n[0], n[1] = 0, Sk
    sc = 1.0 / math.sqrt(D)
    kw = dict(scale=sc, causal=causal, keep_mask=m, kv_len=n, score_clamp=clamp, mode=_lib.MODE_FP32)
    o, lse = ctx.attn_fwd(q, k, v, **kw)
    grads = ctx.attn_bwd(q, k, v, o, lse, do, **kw)
    again = ctx.attn_bwd(q, k, v, o, lse, do, **kw)
    want, mags = _reference(q, k, v, do, sc, causal, m, n, clamp)
    # a sum of n fp32 terms: sqrt(n) roundings of 2^-24 and the few behind each term (scores, exponential, delta: 2^-20 of a term);
    # bf16 results are rounded once, and delta comes from a bf16 output
    for name, got, rep, ref, mag in zip(("dq", "dk", "dv"), grads, again, want, mags):
        assert torch.equal(got, rep), name
        tol = 2.0 ** -18 * mag + (2.0 ** -7 * mag if dt == torch.bfloat16 else 0.0)
        assert float((got.double() - ref).abs().max()) <= tol, (name, float((got.double() - ref).abs().max()), tol)
    assert ctx.device_status() == 0


def test_more_pairs_than_one_launch_has_room_for(ctx):
    B, H, S, D = 4, 9, 2048, 64          # 32 key blocks x 2048 rows x 64 columns of fp32: 16 MB a pair, room for 32 of 36: two launches of 18
    g = torch.Generator(device="cuda").manual_seed(6)
    q, k, v, do = (torch.randn((B, H, S, D), generator=g, device="cuda") for _ in range(4))
    kw = dict(causal=True, mode=_lib.MODE_FP32)
    o, lse = ctx.attn_fwd(q, k, v, **kw)
    grads = ctx.attn_bwd(q, k, v, o, lse, do, **kw)
    for b, h in ((0, 0), (1, 8), (2, 0), (3, 4), (3, 5), (3, 8)):       # the last pair of the first launch is (1, 8)
        one = lambda t: t[b:b + 1, h:h + 1]
        want, mags = _reference(one(q), one(k), one(v), one(do), 1.0 / math.sqrt(D), True, None, None, 0.0)
        for name, got, ref, mag in zip(("dq", "dk", "dv"), grads, want, mags):
            assert float((one(got).double() - ref).abs().max()) <= 2.0 ** -18 * mag, name


def test_a_workspace_without_room_for_the_shares(ctx):
    B, H, S, D = 10, 8, 130, 32
    g = torch.Generator(device="cuda").manual_seed(7)
    q, k, v, do = (torch.randn((B, H, S, D), generator=g, device="cuda") for _ in range(4))
    o, lse = ctx.attn_fwd(q, k, v, mode=_lib.MODE_FP32)
    want, mags = _reference(q, k, v, do, 1.0 / math.sqrt(D), False, None, None, 0.0)
    p = ctx._params(q, k, v, o, lse, 1.0 / math.sqrt(D), False, None, None, 0.0, _lib.MODE_FP32)
    need = (4 * B * H * S + 255) // 256 * 256              # the row sums of dO o O alone
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    got = [torch.empty_like(t) for t in (q, k, v)]
    p.workspace, p.workspace_bytes = ws.data_ptr(), need
    for name, t in (("dout", do), ("dq", got[0]), ("dk", got[1]), ("dv", got[2])):
        setattr(p, name, t.data_ptr())
        setattr(p, "do_strides" if name == "dout" else name + "_strides", _lib.Strides(*t.stride()[:3]))
    ctx.check(ctx.lib.ltca_attn_bwd(ctx.handle, C.byref(p)))
    for name, x, ref, mag in zip(("dq", "dk", "dv"), got, want, mags):
        assert float((x.double() - ref).abs().max()) <= 2.0 ** -18 * mag, name


@pytest.mark.parametrize("B,S,E,H,W", [(2, 32, 32, 4, 32), (3, 31, 24, 2, 30), (2, 5, 8, 2, 64), (2, 1, 16, 1, 9), (2, 33, 16, 2, 16)])
def test_module_backward_that_forms_the_gradient_at_the_context(ctx, B, S, E, H, W):
    """dO = dy Wo^T formed inside the attention backward (up to 32 keys; 33: a product of its own) gives the gradients of the
    module in 64 bits."""
    g = torch.Generator(device="cuda").manual_seed(8)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, dy = rand(B * S, E), rand(B * S, E)
    w = [rand(E, H * W) / math.sqrt(E) for _ in range(3)] + [rand(H * W, E) / math.sqrt(H * W)]
    sc = 1.0 / math.sqrt(W)
    got = ctx.tsa_bwd(x, *w, dy, B, S, H, W, scale=sc, causal=True, time_major=False, mode=_lib.MODE_FP32)
    xd, dyd = x.double(), dy.double()
    leaves = [t.double().requires_grad_() for t in w]
    heads = lambda t: t.view(B, S, H, W).transpose(1, 2)
    q, k, v = (heads(xd @ t) for t in leaves[:3])
    s = (q @ k.transpose(-1, -2) * sc).masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), -math.inf)
    out = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B * S, H * W) @ leaves[3]
    want = torch.autograd.grad((out * dyd).sum(), leaves)
    named = got if isinstance(got, dict) else dict(zip(("dx", "dwq", "dwk", "dwv", "dwo"), got))
    for name, ref in zip(("dwq", "dwk", "dwv", "dwo"), want):
        # chains of at most 64 + 96 + 64 fp32 terms of magnitude about 1
        assert float((named[name].double() - ref).abs().max()) <= 2.0 ** -16 * float(ref.abs().max()) + 1e-6, name
