"""Which exact backward calls ask for room for dQ's shares: those that the one-pass kernel takes, launch by launch.  And a call that has
less room takes more launches, or the two kernels, for the same gradients."""
import ctypes as C
import math

import pytest
import torch

from cuda_ltc_b200 import _lib


def _align(n):
    return (n + 255) // 256 * 256


def _shares(B, H, Sq, Sk, D, causal=False):
    """Bytes that the answer to a size query holds beyond the rows' delta."""
    lib = _lib.load()
    p = _lib.AttnParams()
    p.B, p.H, p.Sq, p.Sk, p.D = B, H, Sq, Sk, D
    p.dtype, p.mode, p.causal, p.scale = _lib.LTCA_F32, _lib.MODE_FP32, int(causal), 1.0
    need = C.c_size_t(0)
    assert lib.ltca_attn_workspace_bytes(C.byref(p), 1, C.byref(need)) == 0
    return need.value - _align(4 * B * H * Sq)


def _one(Sq, Sk, D):
    return (Sk + 63) // 64 * Sq * ((D + 3) // 4 * 4) * 4


@pytest.mark.parametrize("B,H,Sq,Sk,D,causal,pairs", [
    (64, 8, 64, 64, 32, False, 0),             # one block of keys: dQ is written where it belongs
    (4, 4, 512, 512, 32, False, 16),           # 128 CTAs on 148 SMs
    (1, 1, 2048, 2048, 64, False, 0),          # 32 CTAs: the two kernels
    (1, 28, 3000, 128, 64, False, 0),          # 56 CTAs that walk 3000 queries: the two kernels, which deal them out
    (1, 28, 3000, 128, 64, True, 28),          # ... of which the last 128 see a key
    (1, 28, 300, 128, 64, False, 28),
    (1, 42, 3000, 128, 64, False, 42),         # 84 CTAs
    (1, 1, 4096, 4096, 32, False, 0),
    (64, 8, 512, 512, 64, False, 512),         # all pairs at once, the most room there is
    (1, 8, 6000, 6000, 32, False, 4),          # seven pairs fit: two launches of four, a wave each, not 1.1 waves and the rest
    (1, 8, 6000, 6000, 32, True, 7),           # ... which are no shorter where both end on the first keys' chain
    (1, 8, 8192, 8192, 64, False, 2),
    (1, 13, 8192, 8192, 64, True, 0),          # seven launches, each as long as the first keys' chain
    (1, 8, 10000, 10000, 64, False, 0),        # one pair a launch: half of the SMs' places
    (1, 8, 12000, 12000, 32, False, 0),
    (1, 8, 12000, 12000, 32, True, 0),
    (1, 8, 12000, 12000, 64, False, 0),        # one pair's shares are more than there is room for
    (65536, 1, 8, 8, 8, False, 0),             # more batches than a grid takes
    (65536, 1, 8, 128, 8, False, 0),
])
def test_room_for_the_shares(B, H, Sq, Sk, D, causal, pairs):
    assert _shares(B, H, Sq, Sk, D, causal) == pairs * _one(Sq, Sk, D)


@pytest.mark.gpu
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("masked", [False, True])
def test_less_room_takes_more_launches(ctx, causal, masked):
    B, H, Sq, Sk, D = 8, 17, 500, 513, 30
    g = torch.Generator(device="cuda").manual_seed(15)
    rand = lambda n: torch.randn((B, H, n, D), generator=g, device="cuda")
    q, k, v, do = rand(Sq), rand(Sk), rand(Sk), rand(Sq)
    m = (torch.rand((B, Sq, Sk), generator=g, device="cuda") > 0.4).float() if masked else None
    o, lse = ctx.attn_fwd(q, k, v, causal=causal, keep_mask=m, mode=_lib.MODE_FP32)
    p = ctx._params(q, k, v, o, lse, 1.0 / math.sqrt(D), causal, m, None, 0.0, _lib.MODE_FP32)
    need = C.c_size_t(0)
    ctx.check(ctx.lib.ltca_attn_workspace_bytes(C.byref(p), 1, C.byref(need)))
    ws = torch.empty(need.value, dtype=torch.uint8, device="cuda")
    delta, one = _align(4 * B * H * Sq), _one(Sq, Sk, D)
    assert need.value >= delta + B * H * one

    def run(nbytes):
        p.workspace, p.workspace_bytes = ws.data_ptr(), nbytes
        got = [torch.full_like(t, math.nan) for t in (q, k, v)]
        p.dout, p.do_strides = do.data_ptr(), _lib.Strides(*do.stride()[:3])
        for name, t in zip(("dq", "dk", "dv"), got):
            setattr(p, name, t.data_ptr())
            setattr(p, name + "_strides", _lib.Strides(*t.stride()[:3]))
        ctx.check(ctx.lib.ltca_attn_bwd(ctx.handle, C.byref(p)))
        return got

    want = run(need.value)
    # two launches of 68 pairs or so, with and without room for the mask's words
    for room in (68 * one, 70 * one + 100, B * H * one - 1):
        for a, b in zip(run(delta + room), want):
            assert torch.equal(a, b)
    # 136 launches of a pair would be slow: the two kernels
    for a, b in zip(run(delta + one), want):
        assert float((a.double() - b.double()).norm()) <= 1e-5 * float(b.double().norm())
    assert ctx.device_status() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("pre_norm", [0, 1])
@pytest.mark.parametrize("masked", [False, True])
def test_module_without_room_for_the_shares(ctx, pre_norm, masked):
    B, S, H, W = 20, 130, 8, 16
    E = H * W
    g = torch.Generator(device="cuda").manual_seed(16)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda")
    x, dy, gamma, beta = rand(B * S, E), rand(B * S, E), 1.0 + 0.1 * rand(E), 0.1 * rand(E)
    w = [rand(E, E) / math.sqrt(E) for _ in range(4)]
    m = (torch.rand((B, S, S), generator=g, device="cuda") > 0.3).float() if masked else None
    if m is not None:
        m.diagonal(dim1=1, dim2=2).fill_(1.0)
    names = ["dx", "dwq", "dwk", "dwv", "dwo", *(["dbq", "dbk", "dbv", "dbo", "dgamma", "dbeta"] if pre_norm else [])]
    p = _lib.TsaParams()
    p.B, p.S, p.E, p.H, p.head_width, p.scale, p.mode = B, S, E, H, W, W ** -0.5, _lib.MODE_FP32
    p.use_residual = p.use_layer_norm = 1
    p.pre_norm = pre_norm
    p.x, p.dy, p.ln_gamma, p.ln_beta = (t.data_ptr() for t in (x, dy, gamma, beta))
    for name, t in zip(("wq", "wk", "wv", "wo"), w):
        setattr(p, name, t.data_ptr())
    p.keep_mask = m.data_ptr() if masked else None
    need = C.c_size_t(0)
    ctx.check(ctx.lib.ltca_tsa_workspace_bytes(C.byref(p), 3, C.byref(need)))
    shares = B * H * _one(S, S, W)
    words = (S + 31) // 32 * S * B * 4

    def run(nbytes):
        ws = torch.full((max(nbytes, 256) + 4096,), 0x55, dtype=torch.uint8, device="cuda")
        p.workspace, p.workspace_bytes = ws.data_ptr(), nbytes
        got = {n: torch.full_like(t, math.nan) for n, t in zip(names, [x, *w, *([gamma] * 6)])}
        for n, t in got.items():
            setattr(p, n, t.data_ptr())
        rc = ctx.lib.ltca_tsa_bwd(ctx.handle, C.byref(p))
        assert bool((ws[nbytes:] == 0x55).all())          # nothing beyond what was given
        return rc, got

    rc, want = run(need.value)
    assert rc == 0
    for room in (need.value - 256, need.value - shares):
        rc, got = run(room)
        assert rc == 0, ctx.lib.ltca_last_error(ctx.handle)
        for n in names:
            # sums of fp32 terms in another order, three products in a row; dbk's terms, as large as those of dk, sum up to 0 (a shift of
            # all keys moves no softmax): 2^-24 sqrt(rows) of the rows' norm
            scale = max(float(want[o].double().norm()) for o in (("dbk", "dbv") if n == "dbk" else (n,)))
            assert float((got[n].double() - want[n].double()).norm()) <= 2e-5 * scale, n
    rc, _ = run(need.value - shares - (2 * words if masked else 0) - 256)
    assert rc == -4                                       # LTCA_ERR_WORKSPACE
    assert ctx.device_status() == 0
