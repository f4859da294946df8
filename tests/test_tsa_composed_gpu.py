"""The reference's form of the module (heads as wide as the model) where it runs on per-head products of the weights
(Wq_h Wk_h^T, Wv_h Wo_h): from four rows per column of x on.  Both sides of that line, ragged lengths, every mask kind and
the calls that share a kept forward, against the fp64 oracle.  Bounds as in tests/test_tsa_golden.py: no result has more
bf16 roundings behind it than on the path through q, k, v and ctx."""
import numpy as np
import pytest

import oracle
from util import rel_l2

MODULE_REL_L2, MODULE_GRAD_REL_L2, MODULE_MAX_ABS = 5e-3, 7e-3, 2.0 ** -7

# B, S, E, H, causal, time_major, mask, mode
CASES = [
    (4, 136, 136, 2, False, True, False, "auto"),       # exactly four rows per column; one tile and a remainder everywhere
    (5, 109, 136, 2, True, False, False, "auto"),       # one row more, odd length
    (4, 135, 136, 2, False, True, False, "auto"),       # just below: q, k, v and ctx
    (9, 33, 72, 3, False, False, True, "bf16"),         # tiles wider than every matrix, dense mask
    (3, 300, 200, 1, True, True, False, "auto"),        # one head; more keys than a row kernel's first form
    (16, 64, 256, 4, False, True, False, "auto"),       # the smallest of a model's sizes
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES)
def test_module_on_products_of_the_weights(case):
    import torch
    import cuda_ltc_b200 as ltc
    from cuda_ltc_b200 import _lib
    B, S, E, H, causal, time_major, use_mask, mode_name = case
    mode = _lib.MODE_AUTO if mode_name == "auto" else _lib.MODE_BF16
    ctx = ltc.Context(0)
    rng = np.random.default_rng(7)
    lim = np.sqrt(3.0 / E)
    x = (0.5 * rng.standard_normal((B * S, E))).astype(np.float32)
    dy = rng.standard_normal((B * S, E)).astype(np.float32)
    wq, wk = (rng.uniform(-lim, lim, (E, H * E)).astype(np.float32) * 0.5 for _ in range(2))
    wv = rng.uniform(-lim, lim, (E, H * E)).astype(np.float32)
    wo = rng.uniform(-lim, lim, (H * E, E)).astype(np.float32)
    m = None
    if use_mask:
        m = (rng.random((B, S, S)) < 0.8).astype(np.float32)
        m[:, np.arange(S), np.arange(S)] = 1.0
    _, y_ref = oracle.tsa_fwd(x, wq, wk, wv, wo, B, S, H, E, 1.0, causal, time_major, True, True, np.ones(E, np.float32),
                              np.zeros(E, np.float32), None, None, None, None, m)
    gref = oracle.tsa_bwd(x, wq, wk, wv, wo, dy, B, S, H, E, 1.0, causal, time_major, None, None, None, m)
    dev = lambda a: None if a is None else torch.from_numpy(a).cuda()
    args = tuple(dev(a) for a in (x, wq, wk, wv, wo))
    kw = dict(scale=1.0, causal=causal, time_major=time_major, mode=mode, keep_mask=dev(m))
    plain = dict(use_residual=False, use_layer_norm=False, **kw)
    y = ctx.tsa_fwd(*args, B, S, H, E, **plain)
    got = ctx.tsa_bwd(*args, dev(dy), B, S, H, E, **kw)
    cache = ctx.tsa_weight_cache(*args, B, S, H, E, mode=mode, causal=causal)
    assert rel_l2(y.cpu().numpy(), y_ref) < MODULE_REL_L2
    assert np.abs(y.cpu().numpy() - y_ref).max() < MODULE_MAX_ABS * max(1.0, np.abs(y_ref).max())
    for name, g, r in zip(("dx", "dwq", "dwk", "dwv", "dwo"), got, gref):
        gh = g.cpu().numpy().astype(np.float64)
        assert rel_l2(gh, r) < MODULE_GRAD_REL_L2, f"{name}: rel-L2 {rel_l2(gh, r)}"
        assert np.abs(gh - r).max() < MODULE_MAX_ABS * max(1.0, np.abs(r).max()), name
    # a kept forward, twice, and kept weights: the same bits
    saved = ctx.tsa_saved_buffer(*args, B, S, H, E, mode=mode, causal=causal)
    assert torch.equal(y, ctx.tsa_fwd(*args, B, S, H, E, saved=saved, weight_cache=(cache, False), **plain))
    for valid in (True, True):
        kept = ctx.tsa_bwd(*args, dev(dy), B, S, H, E, saved=saved, reuse_forward=True, weight_cache=(cache, valid), **kw)
        for a, b in zip(got, kept):
            assert torch.equal(a, b)
    # kept weights also serve other numbers of rows
    few = ctx.tsa_weight_cache(x_few := args[0][:S], *args[1:], 1, S, H, E, mode=mode, causal=causal)
    fkw = dict(plain, keep_mask=None if m is None else dev(m[:1]))
    ctx.tsa_fwd(x_few, *args[1:], 1, S, H, E, weight_cache=(few, False), **fkw)
    assert torch.equal(y, ctx.tsa_fwd(*args, B, S, H, E, weight_cache=(few, True), **plain))
    # biases go through q, k and v, in blocks sized without them
    bias = [(0.1 * rng.standard_normal(H * E)).astype(np.float32) for _ in range(3)]
    bkw = dict(bq=dev(bias[0]), bk=dev(bias[1]), bv=dev(bias[2]))
    _, yb_ref = oracle.tsa_fwd(x, wq, wk, wv, wo, B, S, H, E, 1.0, causal, time_major, True, True, np.ones(E, np.float32),
                               np.zeros(E, np.float32), *bias, None, m)
    yb = ctx.tsa_fwd(*args, B, S, H, E, saved=saved, **bkw, **plain)
    assert rel_l2(yb.cpu().numpy(), yb_ref) < MODULE_REL_L2
    torch.cuda.synchronize()
    assert ctx.device_status() == 0


@pytest.mark.gpu
def test_bias_gradients_without_biases():
    """The FlashAttention form asks for bias gradients whether it has biases or not."""
    import torch
    import cuda_ltc_b200 as ltc
    from cuda_ltc_b200 import _lib
    B, S, E = 8, 140, 200
    ctx = ltc.Context(0)
    rng = np.random.default_rng(9)
    lim = np.sqrt(3.0 / E)
    x, dy = ((0.5 * rng.standard_normal((B * S, E))).astype(np.float32) for _ in range(2))
    w = [rng.uniform(-lim, lim, (E, E)).astype(np.float32) for _ in range(4)]
    dev = lambda a: torch.from_numpy(a).cuda()
    args = (dev(x), *(dev(a) for a in w))
    one, zero = torch.ones(E, device="cuda"), torch.zeros(E, device="cuda")
    kw = dict(gamma=one, beta=zero, mode=_lib.MODE_AUTO)
    got = ctx.fa_bwd(*args, dev(dy), B, S, 1, E, **kw)
    # zero biases take the path through q, k and v
    ref = ctx.fa_bwd(*args, dev(dy), B, S, 1, E, biases=(zero, zero, zero, zero), **kw)
    out, out_ref = (ctx.fa_fwd(*args, B, S, 1, E, biases=b, **kw) for b in ((None,) * 4, (zero, zero, zero, zero)))
    assert rel_l2(out.cpu().numpy(), out_ref.cpu().numpy()) < MODULE_REL_L2
    for name in ("dx", "dwq", "dwk", "dwv", "dwo", "dbq", "dbv", "dbo", "dgamma", "dbeta"):
        assert rel_l2(got[name].cpu().numpy(), ref[name].cpu().numpy()) < 2 * MODULE_GRAD_REL_L2, name
    # (dbk: the terms of a key bias's gradient cancel, both are rounding errors of sums of |dS| |q|)
    assert got["dbk"].abs().max() < 0.05 * ref["dbq"].abs().max()
    torch.cuda.synchronize()
    assert ctx.device_status() == 0


def _bias_gradients(ctx, p, dy, saved, bias, HW, E):
    """dbq, dbk, dbv, dbo and dwq of a backward that reuses `saved`, `bias` (or None) given to the call."""
    import ctypes as C
    import torch
    out = {n: torch.full((HW if n != "dbo" else E,), float("nan"), device="cuda") for n in ("dbq", "dbk", "dbv", "dbo")}
    dw = {n: torch.empty(HW * E, device="cuda") for n in ("dwq", "dwk", "dwv", "dwo")}
    for n, t in (*out.items(), *dw.items()):
        setattr(p, n, t.data_ptr())
    for n in ("bq", "bk", "bv"):
        setattr(p, n, bias[n].data_ptr() if bias else None)
    p.dy, p.saved, p.saved_bytes, p.reuse_forward = dy.data_ptr(), saved.data_ptr(), saved.numel(), 1
    need = C.c_size_t(0)
    ctx.check(ctx.lib.ltca_tsa_workspace_bytes(C.byref(p), 2, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), need.value
    ctx.check(ctx.lib.ltca_tsa_bwd_weights(ctx.handle, C.byref(p)))
    torch.cuda.synchronize()
    return [*out.values(), dw["dwq"]]


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(4, 136, 136, 2, False, True), (8, 140, 200, 1, True, False), (4, 135, 136, 2, False, True)])
def test_kept_forward_is_read_in_the_form_it_was_written(case):
    """The backward that reuses a kept forward needs no biases: whether it is given them or not, it takes the block as the
    forward wrote it, by another context and from a copy of the block too."""
    import torch
    import cuda_ltc_b200 as ltc
    from cuda_ltc_b200 import _lib
    B, S, E, H, causal, time_major = case
    ctx, other = ltc.Context(0), ltc.Context(0)
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    lim = (3.0 / E) ** 0.5
    x, dy = 0.5 * rnd(B * S, E), rnd(B * S, E)
    w = [lim * 0.5 * rnd(E, H * E) for _ in range(3)] + [lim * 0.5 * rnd(H * E, E)]
    biases = {n: 0.3 * rnd(H * E) for n in ("bq", "bk", "bv")}
    kw = dict(causal=causal, time_major=time_major)
    plain = dict(use_residual=False, use_layer_norm=False, **kw)
    saved = ctx.tsa_saved_buffer(x, *w, B, S, H, E, causal=causal)
    want = {}
    for name, b in (("biased", biases), ("unbiased", {})):
        want[name] = ctx.tsa_bwd(x, *w, dy, B, S, H, E, **kw, **b)                # recomputes the forward
    assert rel_l2(want["biased"][1].cpu().numpy(), want["unbiased"][1].cpu().numpy()) > 0.05
    for name, b in (("biased", biases), ("unbiased", {}), ("biased", biases)):
        ctx.tsa_fwd(x, *w, B, S, H, E, saved=saved, **plain, **b)
        torch.cuda.synchronize()
        for c, block in ((ctx, saved), (other, saved), (ctx, saved.clone())):
            for given in ({}, biases):
                got = c.tsa_bwd(x, *w, dy, B, S, H, E, saved=block, reuse_forward=True, **kw, **given)
                torch.cuda.synchronize()
                for a, r in zip(got, want[name]):
                    assert torch.equal(a, r), (name, bool(given))
        p = ctx._tsa_sizes(x, *w, B, S, H, E, _lib.MODE_AUTO, causal)
        p.time_major = int(time_major)
        p.x, p.wq, p.wk, p.wv, p.wo = (t.data_ptr() for t in (x, *w))
        sums = [_bias_gradients(ctx, p, dy, saved, given, H * E, E) for given in (None, biases)]
        for a, r in zip(*sums):
            assert torch.isfinite(a).all() and torch.equal(a, r), name
        assert rel_l2(sums[0][3].cpu().numpy(), dy.sum(0, dtype=torch.float64).cpu().numpy()) < 1e-5
        assert torch.equal(sums[0][4].view(E, H * E), want[name][1])
    # a backward that recomputes into the block leaves it in its own call's form
    got = ctx.tsa_bwd(x, *w, dy, B, S, H, E, saved=saved, **kw)
    again = ctx.tsa_bwd(x, *w, dy, B, S, H, E, saved=saved, reuse_forward=True, **kw, **biases)
    for a, b, r in zip(got, again, want["unbiased"]):
        assert torch.equal(a, r) and torch.equal(b, r)
    torch.cuda.synchronize()
    assert ctx.device_status() == 0 and other.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("case", [(4, 136, 136, 2), (16, 64, 256, 4)])
def test_results_that_start_off_a_16_byte_boundary(case):
    """Results that TMA cannot store or add to: a product of their own for each of the weights, and dx added to in place."""
    import ctypes as C
    import torch
    import cuda_ltc_b200 as ltc
    from cuda_ltc_b200 import _lib
    B, S, E, H = case
    ctx = ltc.Context(0)
    g = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")
    lim = (3.0 / E) ** 0.5
    x, dy = 0.5 * rnd(B * S, E), rnd(B * S, E)
    w = [lim * 0.5 * rnd(E, H * E) for _ in range(3)] + [lim * 0.5 * rnd(H * E, E)]
    want = ctx.tsa_bwd(x, *w, dy, B, S, H, E)
    p = ctx._tsa_sizes(x, *w, B, S, H, E, _lib.MODE_AUTO, False)
    p.time_major = 1
    p.x, p.wq, p.wk, p.wv, p.wo, p.dy = (t.data_ptr() for t in (x, *w, dy))
    got = [torch.full((t.numel() + 2,), float("nan"), device="cuda") for t in want]
    for n, t in zip(("dx", "dwq", "dwk", "dwv", "dwo"), got):
        setattr(p, n, t.data_ptr() + 4)
    need = C.c_size_t(0)
    ctx.check(ctx.lib.ltca_tsa_workspace_bytes(C.byref(p), 2, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), need.value
    ctx.check(ctx.lib.ltca_tsa_bwd(ctx.handle, C.byref(p)))
    torch.cuda.synchronize()
    for a, r in zip(got, want):
        # the same products; sums of fp32 in another order at most
        assert rel_l2(a[1:-1].cpu().numpy(), r.flatten().cpu().numpy()) < 1e-6
        assert torch.isnan(a[0]) and torch.isnan(a[-1])
    assert ctx.device_status() == 0
