"""Dense masks packed into words (attn_mask.cu) at the edges of the 32 x 32 blocks, in every tensor-pipe kernel that reads
them, and the same bits from calls whose workspace has no room for the words."""
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


@pytest.mark.parametrize("shape", [(2, 2, 1, 1, 16), (1, 3, 31, 33, 32), (2, 80, 70, 97, 64), (1, 2, 129, 65, 128),
                                   # one pass over more than two key blocks: by words, and without room for them on the mask as it is
                                   (3, 40, 70, 161, 32), (2, 40, 130, 257, 16), (3, 20, 65, 190, 64)])
@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
def test_exact_backward_in_a_workspace_sized_without_the_mask(ctx, shape, dt):
    B, H, Sq, Sk, D = shape
    q, k, v, do = (torch.from_numpy(randn((B, H, n, D), 80 + i)).cuda().to(dt) for i, n in enumerate((Sq, Sk, Sk, Sq)))
    m = torch.from_numpy(keep_mask(B, Sq, Sk, 3, 0.6)).cuda()
    o, lse = ctx.attn_fwd(q, k, v, keep_mask=m, mode=_lib.MODE_FP32)
    want = ctx.attn_bwd(q, k, v, o, lse, do, keep_mask=m, mode=_lib.MODE_FP32)
    p = ctx._params(q, k, v, o, lse, 1.0 / math.sqrt(D), False, None, None, 0.0, _lib.MODE_FP32)
    need = C.c_size_t(0)
    ctx.check(ctx.lib.ltca_attn_workspace_bytes(C.byref(p), 1, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    got = [torch.empty_like(t) for t in (q, k, v)]
    p.keep_mask, p.workspace, p.workspace_bytes = m.data_ptr(), ws.data_ptr(), need.value
    for name, t in (("dout", do), ("dq", got[0]), ("dk", got[1]), ("dv", got[2])):
        setattr(p, name, t.data_ptr())
        setattr(p, "do_strides" if name == "dout" else name + "_strides", _lib.Strides(*t.stride()[:3]))
    ctx.check(ctx.lib.ltca_attn_bwd(ctx.handle, C.byref(p)))
    for a, b in zip(got, want):
        assert torch.equal(a, b)


# exact and tensor-pipe pipelines; both forms of the module
@pytest.mark.parametrize("shape", [(3, 21, 32, 2, 16), (2, 85, 128, 2, 64)])
@pytest.mark.parametrize("pre_norm", [0, 1])
def test_module_in_a_workspace_sized_without_the_mask(ctx, shape, pre_norm):
    B, S, E, H, W = shape
    r = lambda *n, amp=1.0: torch.from_numpy(randn(n, 90 + len(n) + n[0], amp)).cuda()
    x, dy = r(B * S, E), r(B * S, E).roll(1, 0)
    w = [r(E, H * W, amp=E ** -0.5) for _ in range(3)] + [r(H * W, E, amp=E ** -0.5)]
    gamma, beta = 1.0 + 0.1 * r(E), 0.1 * r(E)
    m = torch.from_numpy(keep_mask(B, S, S, 3, 0.6)).cuda()
    if pre_norm:
        out = ctx.fa_fwd(x, *w, B, S, H, W, gamma=gamma, beta=beta, keep_mask=m, dropout_prob=0.1, dropout_seed=3)
        g = ctx.fa_bwd(x, *w, dy, B, S, H, W, gamma=gamma, beta=beta, keep_mask=m, dropout_prob=0.1, dropout_seed=3)
    else:
        kw = dict(scale=W ** -0.5, time_major=False, keep_mask=m)
        out = ctx.tsa_fwd(x, *w, B, S, H, W, gamma=gamma, beta=beta, **kw)
        g = dict(zip(("dx", "dwq", "dwk", "dwv", "dwo"), ctx.tsa_bwd(x, *w, dy, B, S, H, W, **kw)))
    got = {n: torch.empty_like(t) for n, t in g.items()}
    y = torch.empty_like(out)
    p = _lib.TsaParams()
    p.B, p.S, p.E, p.H, p.head_width, p.scale, p.mode = B, S, E, H, W, W ** -0.5, _lib.MODE_AUTO
    p.use_residual = p.use_layer_norm = 1
    p.x, p.out, p.dy, p.ln_gamma, p.ln_beta = (t.data_ptr() for t in (x, y, dy, gamma, beta))
    for name, t in [*zip(("wq", "wk", "wv", "wo"), w), *got.items()]:
        setattr(p, name, t.data_ptr())
    if pre_norm:
        p.pre_norm, p.score_clamp, p.dropout_prob, p.dropout_seed = 1, 10.0, 0.1, 3
    need = C.c_size_t(0)
    for which, call in ((0, ctx.lib.ltca_tsa_fwd), (3, ctx.lib.ltca_tsa_bwd)):
        p.keep_mask = None
        ctx.check(ctx.lib.ltca_tsa_workspace_bytes(C.byref(p), which, C.byref(need)))
        ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
        p.keep_mask, p.workspace, p.workspace_bytes = m.data_ptr(), ws.data_ptr(), need.value
        ctx.check(call(ctx.handle, C.byref(p)))
    torch.cuda.synchronize()
    assert torch.equal(y, out)
    for n, t in g.items():
        assert torch.equal(got[n], t), n
