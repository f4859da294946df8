"""LayerNorm rows of every width that stays in a warp's registers (multiples of 128 up to 1024) and of one beyond: the end of the
module's forward and the start of the FlashAttention form's backward, against the oracle.  Bound: fp32 sums of up to 1152
terms, 1152 x 2^-24 = 7e-5, in a chain of three products."""
import numpy as np
import pytest

import oracle
from test_fa_module import make


@pytest.mark.gpu
@pytest.mark.parametrize("width", [128 * n for n in range(1, 10)])
def test_layer_norm_rows(ctx, width):
    import torch
    from cuda_ltc_b200 import _lib
    B, S, E, D = 1, 11, width, 64
    H = E // D
    x, dy, wq, wk, wv, wo, biases, gamma, beta, _ = make(B, S, E, H, D, 5, False)
    dev = lambda a: torch.from_numpy(a).cuda()
    args = tuple(dev(a) for a in (x, wq, wk, wv, wo))
    ref, _ = oracle.tsa_fwd(x, wq, wk, wv, wo, B, S, H, D, D ** -0.5, False, False, True, True, gamma, beta, None, None, None,
                            biases[3], None)
    got = ctx.tsa_fwd(*args, B, S, H, D, scale=D ** -0.5, time_major=False, gamma=dev(gamma), beta=dev(beta), bo=dev(biases[3]),
                      mode=_lib.MODE_FP32)
    assert np.abs(got.cpu().numpy() - ref).max() < 2e-4 * max(1.0, np.abs(ref).max())
    for residual in (True, False):
        kw = dict(gamma=gamma, beta=beta, use_residual=residual)
        gref = oracle.fa_bwd(x, wq, wk, wv, wo, dy, B, S, H, D, biases=biases, **kw)
        kw.update(gamma=dev(gamma), beta=dev(beta))
        grads = ctx.fa_bwd(*args, dev(dy), B, S, H, D, biases=tuple(dev(b) for b in biases), mode=_lib.MODE_FP32, **kw)
        for name in ("dx", "dgamma", "dbeta"):
            assert np.abs(grads[name].cpu().numpy() - gref[name]).max() < 2e-4 * max(1.0, np.abs(gref[name]).max()), name
    assert ctx.device_status() == 0
