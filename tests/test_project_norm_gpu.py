"""The small exact module where a launch does two steps: the end of its forward (projection, residual, LayerNorm) and dQ with
the gradient at the context, at the edges of their ranges and beyond them, against the oracle.  Bound: fp32 sums, as for the
exact module."""
import numpy as np
import pytest

import oracle


# B, S, E, H, W: one row, a ragged last block, E no multiple of a warp, the most columns, the most weights, beyond either, the
# most products, beyond them, the widest context
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 32, 4, 32), (3, 7, 32, 2, 16), (2, 9, 36, 3, 12), (2, 20, 64, 4, 32), (1, 33, 64, 8, 16),
                                   (2, 10, 64, 2, 68),
                                   (2, 8, 68, 2, 16), (64, 65, 32, 2, 16), (64, 64, 32, 4, 48), (61, 64, 48, 4, 40),
                                   (3, 11, 4, 4, 512)])
@pytest.mark.parametrize("norm", [False, True])
def test_projection_residual_norm(shape, norm):
    import torch
    import cuda_ltc_b200 as ltc
    from cuda_ltc_b200 import _lib
    B, S, E, H, W = shape
    ctx = ltc.Context(0)
    rng = np.random.default_rng(3)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, bo, gamma, beta = f(B * S, E), 0.1 * f(E), 1 + 0.1 * f(E), 0.1 * f(E)
    w = [f(E, H * W) * 0.2 for _ in range(3)] + [f(H * W, E) * 0.2]
    ref, _ = oracle.tsa_fwd(x, *w, B, S, H, W, W ** -0.5, False, True, norm, norm, gamma, beta, None, None, None, bo, None)
    dev = lambda a: torch.from_numpy(a).cuda()
    got = ctx.tsa_fwd(dev(x), *(dev(a) for a in w), B, S, H, W, scale=W ** -0.5, time_major=True, use_residual=norm,
                      use_layer_norm=norm, gamma=dev(gamma), beta=dev(beta), bo=dev(bo), mode=_lib.MODE_FP32)
    assert np.abs(got.cpu().numpy() - ref).max() < 2e-5 * max(1.0, np.abs(ref).max())
    assert ctx.device_status() == 0


# B, S, E, H, W, time_major: one row, ragged tiles and widths, the widest of either, tiles of 64 rows, too many rows
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1, 1, 8, 1, 8, True), (3, 17, 32, 2, 12, False), (2, 50, 64, 4, 64, True), (4, 33, 40, 2, 20, True),
                                   (16, 8, 32, 8, 32, False), (40, 8, 32, 4, 32, True), (3, 171, 32, 2, 32, False)])
def test_gradients_from_the_output_gradient(shape):
    import torch
    import cuda_ltc_b200 as ltc
    from cuda_ltc_b200 import _lib
    B, S, E, H, W, tm = shape
    ctx = ltc.Context(0)
    rng = np.random.default_rng(4)
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    x, dy = f(B * S, E), f(B * S, E)
    w = [f(E, H * W) * 0.2 for _ in range(3)] + [f(H * W, E) * 0.2]
    ref = oracle.tsa_bwd(x, *w, dy, B, S, H, W, W ** -0.5, True, tm, None, None, None, None)
    dev = lambda a: torch.from_numpy(a).cuda()
    got = ctx.tsa_bwd(dev(x), *(dev(a) for a in w), dev(dy), B, S, H, W, scale=W ** -0.5, causal=True, time_major=tm,
                      mode=_lib.MODE_FP32)
    for name, g, r in zip(("dx", "dwq", "dwk", "dwv", "dwo"), got, ref):
        assert np.abs(g.cpu().numpy() - r).max() < 2e-5 * max(1.0, np.abs(r).max()), name
    assert ctx.device_status() == 0
