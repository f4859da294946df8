"""The work that a program built on this library has it do, as cases that can be timed and compared.

A case is one call (or one forward and its backward) through :class:`cuda_ltc_b200.Context`.  Kinds:

* ``forward``      attention forward: prefill, policy evaluation
* ``step``         attention forward and its backward: a training step of the core
* ``decode``       one query per sequence over a key/value cache
* ``tsa_forward``  TimeSelfAttention module forward (projections, attention, residual, LayerNorm)
* ``tsa_step``     TimeSelfAttention training step: forward that keeps its intermediates, backward that uses them
* ``fa_step``      FlashAttention module (LayerNorm first, biases, clamp, dropout): forward and backward
"""
import math

import torch

import cuda_ltc_b200 as ltc
from cuda_ltc_b200 import _lib

MODES = {"auto": _lib.MODE_AUTO, "bf16": _lib.MODE_BF16, "split": _lib.MODE_SPLIT, "fp32": _lib.MODE_FP32}
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def _core(kind, B, H, Sq, Sk, D, dtype, mode="auto", causal=False, mask=False, lengths=False, clamp=0.0,
          deterministic=False):
    c = dict(kind=kind, B=B, H=H, Sq=Sq, Sk=Sk, D=D, dtype=dtype, mode=mode, causal=causal, mask=mask,
             lengths=lengths, clamp=clamp)
    if kind == "step":
        c["deterministic"] = deterministic
    return c


def _decode(B, H, cache, D, dtype, lengths=True):
    return dict(kind="decode", B=B, H=H, Sk=cache, D=D, dtype=dtype, lengths=lengths)


def _tsa(kind, B, S, E, H, width, causal, time_major, mode="auto"):
    return dict(kind=kind, B=B, S=S, E=E, H=H, width=width, causal=causal, time_major=time_major, mode=mode)


def _fa(B, S, E, H, width, mask, dropout, mode="auto"):
    return dict(kind="fa_step", B=B, S=S, E=E, H=H, width=width, mask=mask, dropout=dropout, mode=mode)


def listed():
    return [
        # one small forward in fp32, the size of the class's own unit test: nothing but latency
        dict(_core("forward", 2, 4, 64, 64, 32, "f32"), name="forward_small_f32"),
        # prefill of a ragged batch whose lengths are no multiple of a tile: bf16, the wider head
        dict(_core("forward", 4, 16, 1500, 1500, 128, "bf16", causal=True, lengths=True), name="forward_prefill_bf16_d128"),
        # training on medium sequences with the reference's fp32 tensors, bf16-class arithmetic
        dict(_core("step", 32, 8, 256, 256, 64, "f32", causal=True), name="step_f32_d64"),
        # the same where the head is narrower than the tensor-core kernels take: exact fp32 arithmetic, dense mask
        dict(_core("step", 16, 8, 250, 250, 32, "f32", mask=True, clamp=10.0), name="step_exact_f32_d32_masked"),
        # long-sequence training, the benchmark's workload: the largest
        dict(_core("step", 8, 16, 4096, 4096, 64, "bf16", causal=True), name="step_long_bf16"),
        # rollout of many sequences at once over their caches: bound by memory
        dict(_decode(256, 8, 1024, 64, "f32"), name="decode_batch_f32"),
        # a few long conversations: less than one (batch, head) pair per SM
        dict(_decode(3, 8, 4000, 64, "bf16"), name="decode_few_bf16"),
        # a model step of the reference's own tests: hidden 32, 4 heads of the model's width, 32 positions
        dict(_tsa("tsa_step", 8, 32, 32, 4, 32, False, True), name="tsa_small_step"),
        # policy evaluation with the compact module at model width 512
        dict(_tsa("tsa_forward", 32, 256, 512, 8, 64, True, False), name="tsa_forward"),
        # training step of the compact module at the model's batch and sequence length
        dict(_tsa("tsa_step", 64, 512, 512, 8, 64, True, False), name="tsa_step"),
        # training step in the reference's form: every head has the width of the model, scale 1, time-major rows
        dict(_tsa("tsa_step", 32, 256, 512, 8, 512, False, True), name="tsa_reference_form_step"),
        # training step of the FlashAttention module with its mask, clamp, biases and dropout; odd length
        dict(_fa(16, 200, 256, 4, 64, True, 0.1), name="fa_module_step"),
    ]


def _log(rng, lo, hi):
    """A whole number, spread evenly over its logarithm."""
    return min(max(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))), lo), hi)


def _length(rng, lo, hi):
    """A sequence length: every second one is a multiple of 16."""
    n = _log(rng, lo, hi)
    return min(max(16, (n + 8) // 16 * 16), hi) if rng.random() < 0.5 else n


def _draw_once(rng):
    kind = rng.choice(("forward", "forward", "step", "step", "decode", "decode", "tsa_forward", "tsa_step", "fa_step"))
    if kind == "decode":
        return _decode(_log(rng, 1, 512), rng.choice((4, 8, 16)), _length(rng, 64, 8192), rng.choice((32, 64, 64, 128)),
                       rng.choice(("f32", "bf16")), rng.random() < 0.75), 1.1e9, 1e12
    if kind in ("forward", "step"):
        exact = rng.random() < 0.4
        B, H = _log(rng, 1, 64), rng.choice((1, 2, 4, 8, 8, 16))
        causal, lengths = rng.random() < 0.6, rng.random() < 0.25
        det = rng.random() < 0.25
        if exact:   # small sequences, fp32 tensors, head widths of the reference's fixtures, mask and clamp as it has them
            S = _length(rng, 8, 512)
            mask = rng.random() < 0.4
            mode = rng.choice(("auto", "auto", "fp32", "split"))
            return _core(kind, B, H, S, S, rng.choice((16, 32, 32, 64)), "f32", mode, causal and not mask, mask, lengths,
                         10.0 if mask else 0.0, det), 2e8, 6e9
        S = _length(rng, 64, 4096)
        D = rng.choice((64, 64, 128)) if kind == "forward" else 64
        Sk = S
        if kind == "forward" and rng.random() < 0.3:      # a later chunk of a prompt: earlier keys are visible too
            Sk = S + _length(rng, 64, 2048)
        return _core(kind, B, H, S, Sk, D, rng.choice(("bf16", "bf16", "f32")), "auto", causal, False, lengths, 0.0,
                     det), 1e9, (3e11 if kind == "forward" else 9.5e11)
    if kind == "fa_step":
        H = rng.choice((2, 4, 8))
        width = rng.choice((16, 32, 64, 64))
        return _fa(_log(rng, 1, 32), _length(rng, 8, 512), H * width, H, width, rng.random() < 0.7,
                   rng.choice((0.0, 0.1))), 1e9, (3e10 if width == 64 else 6e9)
    H = rng.choice((2, 4, 8))
    if rng.random() < 0.3:           # the reference's form: head width = model width
        E = rng.choice((32, 64, 256, 512))
        return _tsa(kind, _log(rng, 1, 32), _length(rng, 8, 256), E, H, E, False, True), 1e9, (3e11 if E > 128 else 6e9)
    return _tsa(kind, _log(rng, 1, 64), _length(rng, 16, 512), H * 64, H, 64, rng.random() < 0.7, rng.random() < 0.3), 1e9, 3e11


def draw(rng):
    while True:
        c, most_bytes, most_flops = _draw_once(rng)
        w = work(c)
        if w["bytes"] <= most_bytes and w["flops"] <= most_flops:
            return c


_contexts = {}


def _context():
    """A program keeps one context for its device and stream."""
    dev = torch.cuda.current_device()
    if dev not in _contexts:
        _contexts[dev] = ltc.Context(dev)
    return _contexts[dev]


def _rand(g, shape, dtype=torch.float32, amp=1.0):
    return (torch.randn(shape, generator=g, device="cuda") * amp).to(dtype)


def _xavier(g, fan_in, fan_out):
    lim = math.sqrt(6.0 / (fan_in + fan_out))
    return (torch.rand((fan_in, fan_out), generator=g, device="cuda") * 2 - 1) * lim


def _lengths(g, B, Sk):
    return torch.randint(1, Sk + 1, (B,), generator=g, device="cuda", dtype=torch.int32)


def _keep_mask(g, B, S):
    """One in five keys hidden, the diagonal kept."""
    m = (torch.rand((B, S, S), generator=g, device="cuda") > 0.2).float()
    m.diagonal(dim1=1, dim2=2).fill_(1.0)
    return m


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    s = dict(case=c, ctx=_context())
    kind = c["kind"]
    if kind in ("forward", "step", "decode"):
        B, H, Sk, D, dt = c["B"], c["H"], c["Sk"], c["D"], DTYPES[c["dtype"]]
        Sq = c.get("Sq", 1)
        amp = 0.5 if c["dtype"] == "bf16" and kind != "decode" else 1.0
        s["q"] = _rand(g, (B, H, Sq, D), dt, amp)
        s["k"], s["v"] = _rand(g, (B, H, Sk, D), dt, amp), _rand(g, (B, H, Sk, D), dt, amp)
        kw = {}
        if c["lengths"]:
            kw["kv_len"] = _lengths(g, B, Sk)
        if kind != "decode":
            kw.update(causal=c["causal"], score_clamp=c["clamp"], mode=MODES[c["mode"]])
            if c["mask"]:
                kw["keep_mask"] = _keep_mask(g, B, Sk)
        if kind == "step":
            s["dout"] = _rand(g, (B, H, Sq, D), dt, amp)
        s["kw"] = kw
        return s
    B, S, E, H, W = c["B"], c["S"], c["E"], c["H"], c["width"]
    s["x"] = _rand(g, (B * S, E))
    s["w"] = [_xavier(g, E, H * W) for _ in range(3)] + [_xavier(g, H * W, E)]
    s["gamma"], s["beta"] = 1.0 + 0.1 * _rand(g, (E,)), 0.1 * _rand(g, (E,))
    s["shape"] = (B, S, H, W)
    if kind != "tsa_forward":
        s["dy"] = _rand(g, (B * S, E))
    mode = MODES[c["mode"]]
    if kind == "fa_step":
        s["kw"] = dict(biases=tuple(0.1 * _rand(g, (n,)) for n in (H * W, H * W, H * W, E)), gamma=s["gamma"], beta=s["beta"],
                       keep_mask=_keep_mask(g, B, S) if c["mask"] else None, dropout_prob=c["dropout"],
                       dropout_seed=int(seed), mode=mode)
        return s
    # compact heads take 1/sqrt(width); the reference passes 1
    s["kw"] = dict(scale=1.0 if W == E else 1.0 / math.sqrt(W), causal=c["causal"], time_major=c["time_major"], mode=mode)
    if kind == "tsa_step":
        s["saved"] = s["ctx"].tsa_saved_buffer(s["x"], *s["w"], *s["shape"], mode=mode, causal=c["causal"])
    return s


def run(s):
    kind, ctx, kw = s["case"]["kind"], s["ctx"], s["kw"]
    if kind == "forward":
        return ctx.attn_fwd(s["q"], s["k"], s["v"], **kw)
    if kind == "step":
        q, k, v = s["q"], s["k"], s["v"]
        o, lse = ctx.attn_fwd(q, k, v, **kw)
        return (o, lse, *ctx.attn_bwd(q, k, v, o, lse, s["dout"], deterministic=s["case"]["deterministic"], **kw))
    if kind == "decode":
        return ctx.attn_decode(s["q"], s["k"], s["v"], **kw)
    if kind == "tsa_forward":
        return ctx.tsa_fwd(s["x"], *s["w"], *s["shape"], gamma=s["gamma"], beta=s["beta"], **kw)
    if kind == "tsa_step":
        out = ctx.tsa_fwd(s["x"], *s["w"], *s["shape"], gamma=s["gamma"], beta=s["beta"], saved=s["saved"], **kw)
        return (out, *ctx.tsa_bwd(s["x"], *s["w"], s["dy"], *s["shape"], saved=s["saved"], reuse_forward=True, **kw))
    out = ctx.fa_fwd(s["x"], *s["w"], *s["shape"], **kw)
    return out, ctx.fa_bwd(s["x"], *s["w"], s["dy"], *s["shape"], **kw)


def work(case):
    """Every operand once; 2 FLOP per multiply-add of the products; half of the scores under a causal mask; lengths that
    are uniform in 1 .. Sk count half."""
    c = case
    kind = c["kind"]
    if kind in ("forward", "step", "decode"):
        B, H, Sk, D, es = c["B"], c["H"], c["Sk"], c["D"], 2 if c["dtype"] == "bf16" else 4
        Sq = c.get("Sq", 1)
        share = (Sk + 1) / (2.0 * Sk) if c["lengths"] else 1.0
        scores = B * H * Sq * Sk * share
        if c.get("causal"):
            scores *= 1.0 - (Sq - 1) / (2.0 * Sk)
        q, kv = B * H * Sq * D * es, 2 * B * H * Sk * D * es * share
        extra = B * Sq * Sk * 4 if c.get("mask") else 0
        lse = B * H * Sq * 4
        if kind != "step":
            return dict(bytes=2 * q + kv + lse + extra, flops=4.0 * scores * D)
        # forward: q, k, v -> o, lse; backward: q, k, v, o, dout, lse -> dq, dk, dv
        grads = 2 * B * H * Sk * D * es
        return dict(bytes=6 * q + 2 * kv + grads + 2 * lse + 2 * extra, flops=14.0 * scores * D)
    B, S, E, H, W = c["B"], c["S"], c["E"], c["H"], c["width"]
    rows, HW = B * S, H * W
    scores = B * H * S * S * (0.5 * (S + 1) / S if c.get("causal") else 1.0)
    x, w = rows * E * 4, 4 * E * HW * 4
    mask = B * S * S * 4 if c.get("mask") else 0
    fwd_flops = 8.0 * rows * E * HW + 4.0 * scores * W
    if kind == "tsa_forward":
        return dict(bytes=2 * x + w, flops=fwd_flops)
    bwd_flops = 16.0 * rows * E * HW + 10.0 * scores * W
    recomputed = 6.0 * rows * E * HW if kind == "fa_step" else 0.0     # nothing is kept between the two calls
    return dict(bytes=5 * x + 3 * w + 2 * mask, flops=fwd_flops + bwd_flops + recomputed)


def tolerance(case):
    c = case
    kind, mode = c["kind"], c["mode"] if "mode" in c else "fp32"
    if kind in ("forward", "step", "decode"):
        if c["dtype"] == "bf16":
            return {"rel": 1e-2}                 # operands, probabilities and results in bf16
        if kind == "decode" or mode == "fp32":
            return {"rel": 1e-5}                 # fp32 sums
        if mode == "split":
            return {"rel": 5e-5}                 # two bf16 terms per operand: 16 bits, several products in a row
        if c["D"] in (64, 128):
            return {"rel": 1e-2}                 # fp32 tensors, products of bf16 operands
        return {"rel": 1e-5}
    if c["width"] == 64 and c["width"] == c["E"]:
        return {"rel": 2e-2}                     # unscaled scores of bf16 operands: their rounding reaches the exponent
    if c["width"] == 64 or c["width"] > 128:
        return {"rel": 1e-2}                     # chained products of bf16 operands
    return {"rel": 2e-5}                         # fp32 sums, several products in a row
