"""Strides of the tensor-pipe backward's results.  fp32 storage takes any multiple of 16 bytes, backward ones included, and bf16
storage takes them for dQ unless the result is asked for bit for bit; a layout changes no bit of an fp32 result, and what lies between
the rows of one stays as it was."""
import ctypes as C
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu

D = 64
CANARY = 1e30


class _Layout:
    """A [B, H, S, 64] result somewhere in a buffer of its own: `pitch` floats a row, axes in `flips` stored backwards."""

    def __init__(self, B, H, S, dtype, pitch=D, heads_inside=False, flips=()):
        shape = (B, S, H, pitch) if heads_inside else (B, H, S, pitch)
        self.buf = torch.full(shape, CANARY, device="cuda", dtype=dtype)
        self.view = self.buf.transpose(1, 2) if heads_inside else self.buf
        self.flips = flips
        st, at = list(self.view.stride()[:3]), 0
        for axis in flips:
            at += (self.view.shape[axis] - 1) * st[axis]
            st[axis] = -st[axis]
        self.ptr, self.strides = self.buf.data_ptr() + at * self.buf.element_size(), _lib.Strides(*st)

    def result(self):
        t = self.view.flip(self.flips) if self.flips else self.view
        assert bool((t[..., D:] == torch.tensor(CANARY, dtype=t.dtype, device="cuda")).all())
        return t[..., :D]


LAYOUTS = [
    dict(),
    dict(pitch=68),
    dict(heads_inside=True),
    dict(flips=(2,)),
    dict(flips=(1,), pitch=72),
    dict(flips=(0, 1, 2), heads_inside=True),
]


def _backward(ctx, q, k, v, o, lse, do, causal, det, layouts):
    p = ctx._params(q, k, v, o, lse, 1.0 / math.sqrt(D), causal, None, None, 0.0, _lib.MODE_BF16)
    p.bwd_deterministic = int(det)
    need = C.c_size_t(0)
    ctx.check(ctx.lib.ltca_attn_workspace_bytes(C.byref(p), 1, C.byref(need)))
    ws = torch.empty(max(need.value, 256), dtype=torch.uint8, device="cuda")
    p.workspace, p.workspace_bytes = ws.data_ptr(), need.value
    p.dout, p.do_strides = do.data_ptr(), _lib.Strides(*do.stride()[:3])
    for name, l in zip(("dq", "dk", "dv"), layouts):
        setattr(p, name, l.ptr)
        setattr(p, name + "_strides", l.strides)
    ctx.check(ctx.lib.ltca_attn_bwd(ctx.handle, C.byref(p)))
    return [l.result() for l in layouts]


def _inputs(ctx, B, H, Sq, Sk, causal, dtype):
    g = torch.Generator(device="cuda").manual_seed(14)
    rand = lambda n: (torch.randn((B, H, n, D), generator=g, device="cuda") * 0.5).to(dtype)
    q, k, v, do = rand(Sq), rand(Sk), rand(Sk), rand(Sq)
    o, lse = ctx.attn_fwd(q, k, v, causal=causal, mode=_lib.MODE_BF16)
    return q, k, v, o, lse, do


@pytest.mark.parametrize("B,H,Sq,Sk,causal", [(2, 3, 130, 257, True), (1, 1, 1, 65, False), (3, 2, 128, 64, True)])
@pytest.mark.parametrize("layout", LAYOUTS[1:])
def test_layouts_of_fp32_gradients(ctx, B, H, Sq, Sk, causal, layout):
    t = _inputs(ctx, B, H, Sq, Sk, causal, torch.float32)
    of = lambda kw: [_Layout(B, H, S, torch.float32, **kw) for S in (Sq, Sk, Sk)]
    want = _backward(ctx, *t, causal, False, of({}))
    for name, a, b in zip(("dq", "dk", "dv"), _backward(ctx, *t, causal, False, of(layout)), want):
        assert torch.equal(a, b), name
    mixed = [_Layout(B, H, S, torch.float32, **kw) for S, kw in zip((Sq, Sk, Sk), (layout, {}, layout))]
    for name, a, b in zip(("dq", "dk", "dv"), _backward(ctx, *t, causal, False, mixed), want):
        assert torch.equal(a, b), name
    assert ctx.device_status() == 0


@pytest.mark.parametrize("flips", [(2,), (0, 1)])
def test_short_bf16_call_with_a_backwards_dq(ctx, flips):
    B, H, S = 2, 4, 128
    t = _inputs(ctx, B, H, S, S, True, torch.bfloat16)
    of = lambda **kw: [_Layout(B, H, S, torch.bfloat16, **kw)] + [_Layout(B, H, S, torch.bfloat16) for _ in range(2)]
    want = _backward(ctx, *t, True, False, of())
    for name, a, b in zip(("dq", "dk", "dv"), _backward(ctx, *t, True, False, of(flips=flips)), want):
        # each within the bf16 mode's bound of the 64-bit gradients (test_bwd_tiles_gpu.py)
        a, b = a.double(), b.double()
        assert bool(((a - b).abs() <= 4e-3 * max(1.0, float(b.abs().max())) + 2.0 ** -7 * b.abs()).all()), name
    assert ctx.device_status() == 0
