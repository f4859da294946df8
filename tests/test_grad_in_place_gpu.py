"""Gradients written over operands: short bf16 calls whose results take the place of K and V, or of Q or dO where the result need not be
the same bit for bit, and fp32 ones, whose operands are packed first, over any."""
import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu


def _run(ctx, B, H, S, dtype, causal, det, places):
    g = torch.Generator(device="cuda").manual_seed(17)
    rand = lambda: (torch.randn((B, H, S, 64), generator=g, device="cuda") * 0.5).bfloat16().to(dtype)
    t = dict(q=rand(), k=rand(), v=rand(), do=rand())
    kw = dict(causal=causal, mode=_lib.MODE_BF16)
    o, lse = ctx.attn_fwd(t["q"], t["k"], t["v"], **kw)
    out = {n: t[places[n]] if n in places else torch.empty_like(t["q"]) for n in ("dq", "dk", "dv")}
    return ctx.attn_bwd(t["q"], t["k"], t["v"], o, lse, t["do"], deterministic=det, **out, **kw)


@pytest.mark.parametrize("B,H,S,causal", [(1, 2, 300, False), (4, 8, 128, True), (3, 5, 200, True)])
@pytest.mark.parametrize("dtype,det,places", [
    (torch.bfloat16, True, dict(dk="k", dv="v")),
    (torch.bfloat16, False, dict(dk="k", dv="v")),
    (torch.bfloat16, False, dict(dq="q")),
    (torch.bfloat16, False, dict(dq="do", dk="k")),
    (torch.float32, False, dict(dq="q", dk="k", dv="v")),
    (torch.float32, False, dict(dq="k", dk="do", dv="q")),
])
def test_results_in_the_place_of_operands(ctx, B, H, S, causal, dtype, det, places):
    want = _run(ctx, B, H, S, dtype, causal, det, {})
    for name, a, b in zip(("dq", "dk", "dv"), _run(ctx, B, H, S, dtype, causal, det, places), want):
        if dtype == torch.float32 or det:
            assert torch.equal(a, b), name
            continue
        # each within the bf16 mode's bound of the 64-bit gradients (test_bwd_tiles_gpu.py)
        a, b = a.double(), b.double()
        assert bool(((a - b).abs() <= 4e-3 * max(1.0, float(b.abs().max())) + 2.0 ** -7 * b.abs()).all()), name
    assert ctx.device_status() == 0
