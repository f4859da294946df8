"""dx and the four weight gradients of a small tensor-pipe module share a launch; with fewer SMs allowed they do not, and every
gradient keeps its bits."""
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,H", [(1, 1, 1), (3, 43, 1), (2, 65, 2), (5, 77, 3), (8, 128, 4), (16, 200, 4)])
def test_one_launch_and_several_give_the_same_bits(ctx, B, S, H):
    E = 64 * H
    g = torch.Generator(device="cuda").manual_seed(11)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, dy = rand(B * S, E), rand(B * S, E)
    w = [rand(E, E) / math.sqrt(E) for _ in range(4)]
    run = lambda: ctx.tsa_bwd(x, *w, dy, B, S, H, 64, scale=0.125, time_major=False, mode=_lib.MODE_BF16)
    one = run()
    try:
        ctx.set_sm_limit(3)
        several = run()
    finally:
        ctx.set_sm_limit(0)
    for name, a, b in zip(("dx", "dwq", "dwk", "dwv", "dwo"), one, several):
        assert torch.equal(a, b), name
    # and they are the gradients: dWo = ctx^T dy has no other kernel's rounding in it but the context's
    xd, dyd = x.double(), dy.double()
    heads = lambda t: t.view(B, S, H, 64).transpose(1, 2)
    q, k, v = (heads(xd @ t.double()) for t in w[:3])
    out = (torch.softmax(q @ k.transpose(-1, -2) * 0.125, -1) @ v).transpose(1, 2).reshape(B * S, E)
    want = out.t() @ dyd
    assert float((one[4].double() - want).norm()) <= 1e-2 * float(want.norm())
    assert ctx.device_status() == 0
