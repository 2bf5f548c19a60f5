"""Timing cases: the work a program built on `flashlinear` gives the library, through its public
Functions. A case is a plain dict:

  mode    "train"       LinearAttention / LinearAttentionSmallVHD (dk != dv), forward + backward
          "forward"     the same Functions without gradients (scoring, encoder passes)
          "normalized"  LinearAttentionNormalized, forward + backward (denominator included)
          "features"    TaylorLinearAttention on raw inputs of dim `dk`, forward + backward
          "resume"      LinearAttentionResumable without gradients, from a running state to the next:
                        chunked prefill (many tokens a call) and decode (one or a few)
  B, H, N, dk, dv       batch, heads, tokens per call, q/k and v head dims
  dtype   "bf16" | "fp16"
  layout  "bhnd": contiguous [B, H, N, D]; "bnhd": the [B, H, N, D] view of a [B, N, H, D] projection

Inputs follow the library's benchmark: q, k = elu(N(0,1)) + 1 (Taylor features resp. raw N(0,1) for the
feature workloads), v and the upstream gradient ~ N(0,1). fp16 inputs have q scaled by 1/sqrt(dk), as
the acceptance tests do, which keeps the unnormalised sums inside fp16's range.
"""
import math

import torch

from flashlinear import LinearAttention, LinearAttentionSmallVHD
from flashy_linear_attention_b200 import (
    LinearAttentionNormalized,
    LinearAttentionResumable,
    TaylorLinearAttention,
)

TAYLOR_FEATURES = 273  # 1 + 16 + 16^2


def _case(mode, B, H, N, dk, dv, dtype="bf16", layout="bhnd", name=None):
    case = {"mode": mode, "B": B, "H": H, "N": N, "dk": dk, "dv": dv, "dtype": dtype, "layout": layout}
    if name is not None:
        case["name"] = name
    return case


def listed():
    return [
        # one decode step of a served batch: 8 sequences x 32 heads, one token each; the running
        # states are nearly all of the traffic
        _case("resume", 8, 32, 1, 128, 128, name="decode_1_token"),
        # chunked prefill: the next 1000 tokens of two sequences in fp16, straight from a projection's
        # [B, N, H, D] layout, a length that is no multiple of the tile
        _case("resume", 2, 32, 1000, 128, 128, dtype="fp16", layout="bnhd", name="prefill_fp16_1000"),
        # the smallest training shape (the acceptance tests' size): launches and host time count
        _case("train", 2, 4, 256, 64, 64, name="train_small"),
        # a head dim whose rows are no multiple of 16 bytes, the longest acceptance-test sequence
        _case("train", 3, 24, 1984, 83, 83, name="train_odd_dim"),
        # ordinary training layer with 64-wide heads
        _case("train", 8, 16, 4096, 64, 64, name="train_d64"),
        # ordinary training layer with 128-wide heads: the headline benchmark
        _case("train", 4, 32, 8192, 128, 128, name="train_d128"),
        # one GPU's share of that layer when its heads are split over eight: few heads, long sequence
        _case("train", 1, 16, 8192, 128, 128, name="train_few_heads"),
        # long context on one GPU: the largest case
        _case("train", 1, 32, 65536, 128, 128, name="train_long"),
        # heads wider than one tensor-core tile on both sides
        _case("train", 2, 16, 4096, 256, 256, name="train_d256"),
        # second-order Taylor features computed by the caller: wide q/k, narrow v
        _case("train", 8, 16, 2048, TAYLOR_FEATURES, 64, name="train_smallv_273"),
        # the same attention from raw 16-dim q, k
        _case("features", 8, 16, 2048, 16, 64, name="train_raw_features"),
        # attention with its denominator
        _case("normalized", 4, 32, 4096, 128, 128, name="train_normalized"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _head_dim(rng):
    """Mostly the usual widths, otherwise anything the acceptance tests draw from."""
    return rng.choice([32, 64, 64, 96, 128, 128]) if rng.random() < 0.7 else rng.randint(16, 127)


def draw(rng):
    most = max(work(c)["bytes"] for c in listed())
    while True:
        mode = rng.choice(["train"] * 4 + ["smallv"] * 2 + ["wide", "forward", "normalized", "features", "resume", "decode"])
        B, H = _log_uniform(rng, 1, 16), rng.choice([1, 2, 4, 8, 12, 16, 24, 32, rng.randint(1, 32)])
        N = 64 * _log_uniform(rng, 1, 1024)
        dtype, layout = "bf16", rng.choice(["bhnd", "bhnd", "bnhd"])
        dk = dv = _head_dim(rng)
        if mode in ("train", "forward", "resume") and rng.random() < 0.2:
            dtype = "fp16"
        if mode == "smallv":
            mode = "train"
            dk = rng.choice([TAYLOR_FEATURES, 96, 128, 160, 256, rng.randint(65, 384)])
            dv = rng.choice([16, 32, 64])
        elif mode == "wide":
            mode, dk = "train", rng.choice([160, 192, 256])
            dv = dk
        elif mode == "normalized":
            dk = dv = rng.choice([32, 64, 96, 128])
        elif mode == "features":
            dk, dv, N = rng.choice([8, 16]), rng.choice([16, 32, 64]), min(N, 8192)
        elif mode == "resume":
            N = _log_uniform(rng, 128, 16384)
        elif mode == "decode":
            mode, N = "resume", _log_uniform(rng, 1, 64)
        case = _case(mode, B, H, N, dk, dv, dtype, layout)
        # no drawn case costs more than the largest listed one (wide heads run well below the rate
        # of 128-wide ones, so they get a quarter of its bytes)
        limit = 0.8 * most if max(dk, dv) <= 128 else 0.2 * most
        if 2e5 < work(case)["bytes"] < limit:
            return case


def _layout(case, t):
    return t.transpose(1, 2).contiguous().transpose(1, 2) if case["layout"] == "bnhd" else t


def _taylor_features(x):
    d = x.shape[-1]
    outer = (x.unsqueeze(-1) * x.unsqueeze(-2)).flatten(-2) / (math.sqrt(2) * math.sqrt(d))
    return torch.cat([torch.ones_like(x[..., :1]), x / math.sqrt(math.sqrt(d)), outer], dim=-1)


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, H, N, dk, dv = (case[x] for x in ("B", "H", "N", "dk", "dv"))
    dtype = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16

    def randn(*shape):
        return torch.randn(*shape, device="cuda", generator=gen)

    def queries(n):
        if case["mode"] == "features":
            return randn(B, H, n, dk)
        if dk == TAYLOR_FEATURES:
            return _taylor_features(randn(B, H, n, 16))
        x = torch.nn.functional.elu(randn(B, H, n, dk)) + 1
        return x

    q = queries(N)
    if dtype == torch.float16:
        q = q / math.sqrt(dk)
    q, k, v = (_layout(case, t.to(dtype)) for t in (q, queries(N), randn(B, H, N, dv)))
    state = {"mode": case["mode"], "q": q, "k": k, "v": v}
    if case["mode"] == "resume":
        # the running state after 256 earlier tokens
        state["s"] = queries(256).transpose(-1, -2) @ randn(B, H, 256, dv)
    elif case["mode"] != "forward":
        state["dy"] = _layout(case, randn(B, H, N, dv).to(dtype))
        for t in (q, k, v):
            t.requires_grad_(True)
    return state


def run(state):
    q, k, v, mode = state["q"], state["k"], state["v"], state["mode"]
    if mode == "resume":
        with torch.no_grad():
            return LinearAttentionResumable.apply(q, k, v, state["s"])
    if mode == "features":
        function = TaylorLinearAttention
    elif mode == "normalized":
        function = LinearAttentionNormalized
    else:
        function = LinearAttention if q.shape[-1] == v.shape[-1] else LinearAttentionSmallVHD
    if mode == "forward":
        with torch.no_grad():
            return function.apply(q, k, v)
    out = function.apply(q, k, v)
    return (out,) + torch.autograd.grad(out, (q, k, v), state["dy"])


def work(case):
    """Forward and backward are two calls, and what they read does not fit a cache between them: q, k,
    v are counted in both. Operations are those of the recurrence (state update and read-out: two
    products forward, five backward)."""
    B, H, N, dk, dv = (case[x] for x in ("B", "H", "N", "dk", "dv"))
    feat = 1 + dk + dk * dk if case["mode"] == "features" else dk
    tokens = B * H * N
    values, products = 2 * dk + 2 * dv, 2
    if case["mode"] in ("train", "normalized", "features"):
        values += (2 * dk + 2 * dv) + (2 * dk + dv)
        products += 5
    if case["mode"] == "normalized":
        values += dv  # the normalised output, which the denominator's gradient reads
    bytes_ = 2 * values * tokens
    if case["mode"] == "resume":
        bytes_ += 2 * 4 * B * H * dk * dv
    return {"bytes": bytes_, "flops": 2 * products * feat * dv * tokens}


def tolerance(case):
    """About four times what the path differs by from an evaluation in 64 bits: operands and results
    rounded to 16 bits, 32-bit sums (measured: bf16 2.4e-3, from raw features 3.3e-3, fp16 2.9e-4,
    largest single value 0.03). With the denominator, dQ and dK are sums of two partly cancelling
    terms, one of them rounded to bf16: measured 7.2e-3, single values up to 0.64."""
    if case["mode"] == "normalized":
        return {"rel": 2.8e-2, "max": 0.99}
    if case["dtype"] == "fp16":
        return {"rel": 1.2e-3, "max": 0.05}
    return {"rel": 1.2e-2, "max": 0.15}
