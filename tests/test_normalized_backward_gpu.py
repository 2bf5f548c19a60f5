"""The denominator's gradient inside the backward kernel (ops.normalized_bwd) against an evaluation in 64 bits,
and the calls that keep the separate kernels."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture
def any_length():
    """Lifts the rule that the kernel only runs above 2048 tokens."""
    from flashy_linear_attention_b200 import _lib, ops

    old = ops.set_debug_flags(_lib.FLA_DEBUG_FORCE_SINGLE_SWEEP)
    yield
    ops.set_debug_flags(old)


def _inputs(B, H, N, D, bnhd):
    gen = torch.Generator(device=DEV).manual_seed(N + D)

    def draw(positive):
        x = torch.randn(B, H, N, D, device=DEV, generator=gen)
        x = (torch.nn.functional.elu(x) + 1 if positive else x).bfloat16()
        return x.transpose(1, 2).contiguous().transpose(1, 2) if bnhd else x

    return draw(True), draw(True), draw(False), draw(False)


# the rule's edges in heads, ragged last chunks (a multiple of 4 tokens), whole and partly used tiles, two rounds;
# one, two and three chunks
@pytest.mark.parametrize("B,H,N,D,bnhd", [(1, 99, 1024, 128, False), (1, 100, 1100, 96, True), (2, 50, 1252, 128, True),
                                          (1, 99, 1024, 64, True), (1, 50, 1024, 56, True), (1, 60, 1156, 40, False), (2, 148, 580, 64, False),
                                          (1, 99, 64, 128, False), (1, 99, 192, 64, True), (1, 100, 324, 96, False)])
def test_against_64_bits(any_length, B, H, N, D, bnhd):
    from flashy_linear_attention_b200 import ops

    q, k, v, dnum = _inputs(B, H, N, D, bnhd)
    # as in earnest: the two parts partly cancel, d_i = -(dnum_i . out_i) with an output of v's size
    dden = -(dnum.float() * v.float().cumsum(2) / torch.arange(1, N + 1, device=DEV).view(1, 1, -1, 1)).sum(-1).view(B * H, N)
    s_last = (k.double().mT @ v.double()).float().view(B * H, D, D)
    got = ops.normalized_bwd(dnum, dden, q, k, v, s_last)
    torch.cuda.synchronize()
    ops.check_status(torch.device(DEV))
    q64, k64, v64, g64 = (t.double() for t in (q, k, v, dnum))
    dp = torch.tril(g64 @ v64.mT + dden.double().view(B, H, N, 1))
    want = dp @ k64, dp.mT @ q64, torch.tril(q64 @ k64.mT).mT @ g64
    # three roundings of 2^-9 / sqrt(3) in norm (operands of scores or state, result); a state's rounding is
    # relative to the product's part alone, which is up to three times the sum it cancels to here
    for name, x, w, t, cancel in zip(("dq", "dk", "dv"), got, want, (q, k, v), (3, 3, 1)):
        assert x.stride() == torch.empty_like(t).stride()
        rel = ((x.double() - w).norm() / w.norm()).item()
        assert rel <= cancel * 2.0**-9 * math.sqrt((1 + 4 + 4) / 3), (name, rel)


def test_is_as_close_to_64_bits_as_the_separate_kernels(any_length):
    from flashy_linear_attention_b200 import LinearAttentionNormalized, ops

    q, k, v, g = _inputs(1, 100, 1024, 128, False)
    tq, tk, tv = (t.detach().requires_grad_(True) for t in (q, k, v))
    grads = torch.autograd.grad(LinearAttentionNormalized.apply(tq, tk, tv), (tq, tk, tv), g)
    out, den, s_final = ops.normalized_fwd(q, k, v, 1e-5, True)
    dnum, dden = ops.normalize_bwd_prepare(g, out, den)
    dq, dk, _ = ops.causal_dot_product_bwd(dnum, q, k, v, s_last=s_final, keep_padded=True)
    ops.normalize_bwd_sweep(q, k, dq, dk, dden)
    q64, k64, v64 = (t[:, :4].double().requires_grad_(True) for t in (q, k, v))
    p = torch.tril(q64 @ k64.mT)
    want = torch.autograd.grad(p @ v64 / (p.sum(-1, keepdim=True) + 1e-5), (q64, k64), g[:, :4].double())
    for name, inside, separate, w in zip(("dq", "dk"), grads, (dq, dk), want):
        err = [((x[:, :4].double() - w).norm() / w.norm()).item() for x in (inside, separate)]
        assert err[0] <= 1.02 * err[1], (name, err)


@pytest.mark.parametrize("shape,dtype", [((1, 98, 1024, 128), torch.bfloat16), ((1, 100, 1024, 84), torch.bfloat16),
                                         ((1, 100, 1022, 128), torch.bfloat16),
                                         ((1, 100, 1024, 128), torch.float16)])
def test_calls_that_keep_the_separate_kernels(any_length, shape, dtype):
    from flashy_linear_attention_b200 import ops

    q = torch.zeros(shape, dtype=dtype, device=DEV)
    B, H, N, D = shape
    dden = torch.zeros(B * H, N, device=DEV)
    s = torch.zeros(B * H, D, D, device=DEV)
    assert ops.normalized_bwd(q, dden, q, q, q, s) is None
    assert ops.normalized_bwd(q, dden, q, q, q, None) is None


@pytest.mark.parametrize("tokens,inside", [(2048, False), (2052, True)])
def test_short_calls_keep_the_separate_kernels(tokens, inside):
    from flashy_linear_attention_b200 import ops

    q = torch.zeros(1, 100, tokens, 128, dtype=torch.bfloat16, device=DEV)
    grads = ops.normalized_bwd(q, torch.zeros(100, tokens, device=DEV), q, q, q, torch.zeros(100, 128, 128, device=DEV))
    assert (grads is not None) == inside
