"""head_dim 128, bf16 results: the probabilities of one 128-key step are taken relative to the maximum of all its keys, so a row's
largest one is exactly 1 and not rounded, wherever in the step its key lies."""
import math

import pytest
import torch

from cuda_ltc_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Sk", [100, 128])
@pytest.mark.parametrize("masked", [False, True])
def test_the_largest_probability_is_exact(ctx, Sk, masked):
    Sq, D = 257, 128
    # key j is 8 e_j, so q's entries are the scores: one key of the first half at 0, one of the second a little above, the rest at -60
    scores = torch.full((Sq, Sk), -60.0, device="cuda")
    rows = torch.arange(Sq, device="cuda")
    scores[rows, rows % 64] = 0.0
    scores[rows, 64 + rows % (Sk - 64)] = torch.linspace(0.05, 3.0, Sq, device="cuda")
    q = torch.zeros((1, 1, Sq, D), device="cuda")
    q[0, 0, :, :Sk] = scores * math.sqrt(D) / 8.0
    k = torch.zeros((1, 1, Sk, D), device="cuda")
    k[0, 0, :, :Sk] = 8.0 * torch.eye(Sk, device="cuda")
    v = torch.zeros((1, 1, Sk, D), device="cuda")
    v[:, :, 64:] = 1.0
    q, k, v = (t.bfloat16() for t in (q, k, v))
    m = torch.ones((1, Sq, Sk), device="cuda") if masked else None
    o, _ = ctx.attn_fwd(q, k, v, keep_mask=m, mode=_lib.MODE_BF16)
    p = torch.softmax(q.double() @ k.double().transpose(-1, -2) / math.sqrt(D), -1)
    want = p @ v.double()                      # in [1/2, 1): half a unit of bf16's last place is 2^-9
    assert float((o.double() - want).abs().max()) <= 2.0 ** -9 + 1e-4     # and fp32 scores, exponentials and sums
    assert ctx.device_status() == 0
