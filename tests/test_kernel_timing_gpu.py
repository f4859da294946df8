"""The three durations of a timed tensor-pipe backward: what each of the forms puts where."""
import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,S,det,one_launch", [
    (torch.float32, 300, False, True),
    (torch.float32, 2000, False, True),
    (torch.bfloat16, 128, False, True),
    (torch.bfloat16, 512, True, True),
    (torch.bfloat16, 2304, False, False),        # fused kernel and dQ's conversion
    (torch.bfloat16, 2304, True, False),         # a kernel for dQ and one for dK and dV
])
def test_stages(ctx, dtype, S, det, one_launch):
    q, k, v, do = (torch.randn((2, 4, S, 64), device="cuda").to(dtype) for _ in range(4))
    o, lse = ctx.attn_fwd(q, k, v, mode=_lib.MODE_BF16)
    ctx.enable_kernel_timing(True)
    try:
        for other in (2304, S):                  # (nothing is left over from a call of another form)
            x = [torch.randn((1, 1, other, 64), device="cuda").bfloat16() for _ in range(4)]
            xo, xl = ctx.attn_fwd(*x[:3], mode=_lib.MODE_BF16)
            ctx.attn_bwd(*x[:3], xo, xl, x[3], mode=_lib.MODE_BF16)
            ctx.attn_bwd(q, k, v, o, lse, do, mode=_lib.MODE_BF16, deterministic=det)
            a, b, c = ctx.last_bwd_kernel_ms()
            assert a > 0.0 and b > 0.0
            assert c == 0.0 if one_launch else c > 0.0
    finally:
        ctx.enable_kernel_timing(False)
