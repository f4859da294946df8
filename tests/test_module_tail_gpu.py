"""The end of the FlashAttention module's backward in two launches: LayerNorm backward with dgamma and dbeta, bias gradients.  Row
widths of every form (scalar up to 128 columns, 16-byte pieces, and one that keeps the launches of its own), rows in one block, in
rounds that end early, and in more than one round of the warps.  Against autograd in 64 bits."""
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1, 8), (3, 7, 2, 20), (5, 33, 3, 32), (2, 61, 2, 64), (9, 250, 1, 128), (3, 50, 4, 96), (2, 70, 5, 128), (2, 9, 8, 128),
         (2, 30, 2, 80)]


@pytest.mark.parametrize("B,S,H,W", CASES)
@pytest.mark.parametrize("residual", [True, False])
def test_layer_norm_and_bias_gradients(ctx, B, S, H, W, residual):
    E = H * W
    g = torch.Generator(device="cuda").manual_seed(12)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, dy = rand(B * S, E), rand(B * S, E)
    w = [rand(E, E) / math.sqrt(E) for _ in range(4)]
    biases = tuple(0.1 * rand(E) for _ in range(4))
    gamma, beta = 1.0 + 0.1 * rand(E), 0.1 * rand(E)
    got = ctx.fa_bwd(x, *w, dy, B, S, H, W, biases=biases, gamma=gamma, beta=beta, use_residual=residual, mode=_lib.MODE_FP32)
    again = ctx.fa_bwd(x, *w, dy, B, S, H, W, biases=biases, gamma=gamma, beta=beta, use_residual=residual, mode=_lib.MODE_FP32)
    leaf = lambda t: t.double().requires_grad_()
    names = ("dx", "dwq", "dwk", "dwv", "dwo", "dbq", "dbk", "dbv", "dbo", "dgamma", "dbeta")
    leaves = [leaf(t) for t in (x, *w, *biases, gamma, beta)]
    xd, wq, wk, wv, wo, bq, bk, bv, bo, gm, bt = leaves
    ln = torch.nn.functional.layer_norm(xd, (E,), gm, bt, 1e-5)
    heads = lambda t: t.view(B, S, H, W).transpose(1, 2)
    q, k, v = (heads(ln @ a + b) for a, b in ((wq, bq), (wk, bk), (wv, bv)))
    s = (q @ k.transpose(-1, -2) / math.sqrt(W)).clamp(max=10.0)
    out = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B * S, E) @ wo + bo + (xd if residual else 0.0)
    want = torch.autograd.grad((out * dy.double()).sum(), leaves)
    mag = max(float(r.abs().max()) for n, r in zip(names, want) if n in ("dbq", "dbk", "dbv"))
    for name, ref in zip(names, want):
        assert torch.equal(got[name], again[name]), name
        # chains of fp32 sums over E, S and the rows, terms of magnitude about 1: some 2^-24 sqrt(rows E) each
        scale = mag if name in ("dbq", "dbk", "dbv") else float(ref.abs().max())
        assert float((got[name].double() - ref).abs().max()) <= 1e-4 * max(1.0, scale), (name, float((got[name].double() - ref).abs().max()))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("B,S,H,dropout", [(16, 200, 4, 0.1), (3, 347, 2, 0.0), (9, 150, 1, 0.0), (8, 160, 3, 0.1)])
def test_sums_over_the_slices_of_split_weight_gradients(ctx, B, S, H, dropout):
    """On the tensor pipe from 1024 rows on the weight gradients' products are split, and the tail adds the slices up: as the products'
    own launch does, which runs where fewer SMs leave no room for the group."""
    E = 64 * H
    g = torch.Generator(device="cuda").manual_seed(18)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    r16 = lambda t: t.bfloat16().float()
    x, dy = rand(B * S, E), r16(rand(B * S, E))
    w = [r16(rand(E, E) / math.sqrt(E)) for _ in range(4)]
    biases = tuple(0.1 * rand(E) for _ in range(4))
    gamma, beta = 1.0 + 0.1 * rand(E), 0.1 * rand(E)
    run = lambda: ctx.fa_bwd(x, *w, dy, B, S, H, 64, biases=biases, gamma=gamma, beta=beta, dropout_prob=dropout, dropout_seed=5, mode=_lib.MODE_BF16)
    one = run()
    try:
        ctx.set_sm_limit(3)
        several = run()
    finally:
        ctx.set_sm_limit(0)
    for name in one:
        assert torch.equal(one[name], several[name]), name
    if dropout:
        assert ctx.device_status() == 0
        return
    names = ("dx", "dwq", "dwk", "dwv", "dwo", "dbq", "dbk", "dbv", "dbo", "dgamma", "dbeta")
    leaves = [t.double().requires_grad_() for t in (x, *w, *biases, gamma, beta)]
    xd, wq, wk, wv, wo, bq, bk, bv, bo, gm, bt = leaves
    ln = torch.nn.functional.layer_norm(xd, (E,), gm, bt, 1e-5)
    heads = lambda t: t.view(B, S, H, 64).transpose(1, 2)
    q, k, v = (heads(ln @ a + b) for a, b in ((wq, bq), (wk, bk), (wv, bv)))
    s = (q @ k.transpose(-1, -2) / 8.0).clamp(max=10.0)
    out = (torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B * S, E) @ wo + bo + xd
    want = dict(zip(names, torch.autograd.grad((out * dy.double()).sum(), leaves)))
    mag = max(float(want[n].abs().max()) for n in ("dbq", "dbk", "dbv"))
    for name, ref in want.items():
        # two stacked roundings to bf16, 2^-7 of the largest magnitude (test_fa_module.py)
        scale = mag if name in ("dbq", "dbk", "dbv") else float(ref.abs().max())
        assert float((one[name].double() - ref).abs().max()) <= 2.0 ** -7 * max(1.0, scale), name
    assert ctx.device_status() == 0
