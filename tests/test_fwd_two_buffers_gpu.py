"""The head_dim 128 forward with bf16 results: one to three key steps of 128, whole and cut, where single rows (and so single
warps) rescale at single steps and the others never do.  Against PyTorch in 64 bits."""
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Sk", [1, 64, 65, 128, 129, 192, 255, 256, 320, 384])
@pytest.mark.parametrize("masked", [False, True])
def test_steps_and_rescales(ctx, Sk, masked):
    B, H, Sq, D = 2, 3, 130, 128
    g = torch.Generator(device="cuda").manual_seed(13)
    rand = lambda n: torch.randn((B, H, n, D), generator=g, device="cuda") * 0.5
    q, k, v = rand(Sq), rand(Sk), rand(Sk)
    # the last key of each step's first half is far above the rest for rows 5, 37 and 129 alone
    q[..., 0], k[..., 0] = 0.0, 0.0
    q[:, :, [5, 37, 129], 0] = 8.0
    peaks = torch.arange(63, max(Sk, 63), 128, device="cuda")
    k[:, :, peaks, 0] = 20.0 + 10.0 * torch.arange(len(peaks), device="cuda")
    q, k, v = (t.bfloat16() for t in (q, k, v))
    m = (torch.rand((B, Sq, Sk), generator=g, device="cuda") > 0.3).float() if masked else None
    o, lse = ctx.attn_fwd(q, k, v, keep_mask=m, mode=_lib.MODE_BF16)
    again, _ = ctx.attn_fwd(q, k, v, keep_mask=m, mode=_lib.MODE_BF16)
    s = q.double() @ k.double().transpose(-1, -2) / math.sqrt(D)
    if masked:
        s = s.masked_fill((m == 0)[:, None], -math.inf)
    p = torch.softmax(s, -1).nan_to_num(0.0)
    want, mag = p @ v.double(), p @ v.double().abs()
    # probabilities and results rounded once each to 8 significant bits; scores up to 60 in fp32 and the exponential's error: 1e-4
    assert torch.equal(o, again)
    assert bool(((o.double() - want).abs() <= (2.0 ** -8 + 1e-4) * mag + 2.0 ** -8 * want.abs() + 1e-6).all())
    ref_lse = torch.logsumexp(s, -1)
    fin = ref_lse.isfinite()
    assert torch.equal(fin, lse.isfinite())
    assert float((lse.double() - ref_lse)[fin].abs().max()) < 2e-3
    assert ctx.device_status() == 0
