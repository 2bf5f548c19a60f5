"""GPU tests of attention with its denominator inside the product kernel (the NORM variant of the
chunk kernel) against the closed form in fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _closed_form(q, k, v, g, eps):
    q, k, v = (t.double().requires_grad_(True) for t in (q, k, v))
    num = torch.tril(q @ k.transpose(-1, -2)) @ v
    den = (q * k.cumsum(-2)).sum(-1, keepdim=True) + eps
    out = num / den
    return (out.detach(), den.detach()) + torch.autograd.grad(out, (q, k, v), g.double())


# one chunk, one and a half, ragged last chunks, the first length of the single sweep (17 chunks) on
# enough heads not to be split; tile widths 64 and 128, whole and partly used; both operand layouts
@pytest.mark.parametrize("single_sweep", [False, True])
@pytest.mark.parametrize("shape", [(1, 2, 64, 128), (2, 2, 192, 64), (1, 3, 320, 96), (1, 2, 704, 128), (2, 1, 576, 32),
                                   (1, 2, 256, 8), (1, 130, 2176, 64), (1, 130, 4096, 128)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
def test_fused_denominator_against_closed_form(shape, layout, single_sweep):
    from flashy_linear_attention_b200 import LinearAttentionNormalized, ops
    from flashy_linear_attention_b200._lib import FLA_DEBUG_FORCE_SINGLE_SWEEP

    B, H, N, d = shape
    if H > 100 and (layout == "bnhd" or single_sweep):
        pytest.skip("the long case runs once")
    gen = torch.Generator(device="cuda").manual_seed(N + d)

    def draw(positive):
        x = torch.randn(B, H, N, d, device="cuda", generator=gen)
        x = (torch.nn.functional.elu(x) + 1 if positive else x).bfloat16()
        return x.transpose(1, 2).contiguous().transpose(1, 2) if layout == "bnhd" else x

    q, k, v, g = draw(True), draw(True), draw(False), draw(False)
    for t in (q, k, v):
        t.requires_grad_(True)
    assert ops.normalized_fused(q, k, v)
    old = ops.set_debug_flags(FLA_DEBUG_FORCE_SINGLE_SWEEP if single_sweep else 0)
    try:
        out = LinearAttentionNormalized.apply(q, k, v, 1e-5)
        grads = torch.autograd.grad(out, (q, k, v), g)
        _, den, _ = ops.normalized_fwd(q.detach(), k.detach(), v.detach(), 1e-5, False)
    finally:
        ops.set_debug_flags(old)
    ops.check_status()
    assert out.is_contiguous()
    heads = slice(0, 2) if H > 100 else slice(None)
    want_out, want_den, *want = _closed_form(*(t.detach()[:, heads] for t in (q, k, v, g)), 1e-5)

    def rel(got, ref):
        return ((got.detach()[:, heads].double() - ref).norm() / ref.norm()).item()

    # fp32 sums of positive terms
    got_den = den.view(B, H, N, 1)[:, heads].double()
    assert ((got_den - want_den).abs() / want_den).max() < 1e-5
    # the bounds of the unfused kernels' test: 1e-2 (16-bit scores, state and result), and twice that
    # for dQ and dK, whose two parts partly cancel
    assert rel(out, want_out) < 1e-2
    assert rel(grads[2], want[2]) < 1e-2
    assert rel(grads[0], want[0]) < 2e-2 and rel(grads[1], want[1]) < 2e-2


def _inputs(B, H, N, d, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = [torch.randn(B, H, N, d, device="cuda", generator=gen) for _ in range(4)]
    return [(torch.nn.functional.elu(t) + 1 if i < 2 else t).bfloat16() for i, t in enumerate(x)]


# few heads and a long sequence: the product is split, the denominator runs in its own kernels, with
# column sums of the segments before (64 and 128 columns are instantiations of their own); last, a whole
# product on too few heads for the fused form
@pytest.mark.parametrize("shape", [(1, 2, 4096, 64), (1, 3, 4160, 128), (1, 2, 4096, 96), (1, 60, 1152, 128)], ids=lambda s: "x".join(map(str, s)))
def test_split_sequences_take_the_separate_kernels(shape):
    from flashy_linear_attention_b200 import LinearAttentionNormalized, ops

    q, k, v, g = _inputs(*shape, seed=shape[-1])
    assert not ops.normalized_fused(q, k, v)
    for t in (q, k, v):
        t.requires_grad_(True)
    out = LinearAttentionNormalized.apply(q, k, v, 1e-5)
    grads = torch.autograd.grad(out, (q, k, v), g)
    den = ops.normalize_fwd(q.detach(), k.detach(), out.detach().clone(), 1e-5).view(*shape[:3], 1)
    ops.check_status()
    want_out, want_den, *want = _closed_form(*(t.detach() for t in (q, k, v, g)), 1e-5)
    assert ((den.double() - want_den).abs() / want_den).max() < 1e-5  # fp32 sums of positive terms

    def rel(got, ref):
        return ((got.detach().double() - ref).norm() / ref.norm()).item()

    assert rel(out, want_out) < 1e-2 and rel(grads[2], want[2]) < 1e-2  # as above
    assert rel(grads[0], want[0]) < 2e-2 and rel(grads[1], want[1]) < 2e-2


@pytest.mark.parametrize("shape", [(1, 130, 1088, 64), (1, 76, 2048, 128), (2, 3, 192, 32)], ids=lambda s: "x".join(map(str, s)))
def test_fused_and_separate_denominators_agree(shape):
    """Both sum in fp32 in different orders and round the same product to 16 bits before they divide: the
    denominators agree to a few 2^-24 of their size times the root of the terms, the outputs to one rounding."""
    from flashy_linear_attention_b200 import ops

    q, k, v, _ = _inputs(*shape, seed=1)
    assert ops.normalized_fused(q, k, v)
    out, den, _ = ops.normalized_fwd(q, k, v, 1e-5, False)
    num = ops.causal_dot_product_fwd(q, k, v)
    den2 = ops.normalize_fwd(q, k, num, 1e-5)  # divides in place
    assert ((den - den2).abs() / den2).max() < 4e-6
    assert ((out.float() - num.float()).abs() <= 2.0**-7 * num.float().abs()).all()
    assert (out != num).float().mean() < 1e-3


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_fused_denominator_keeps_what_comes_before_a_bad_token(d, value):
    """A NaN or infinity in one token's q reaches that token only, in its k the tokens from there on."""
    from flashy_linear_attention_b200 import ops

    q, k, v, _ = _inputs(1, 3, 448, d, seed=2)
    at = 200  # inside the second of four chunks
    clean, den, _ = ops.normalized_fwd(q, k, v, 1e-5, False)
    for which in (0, 1):
        bad = [q.clone(), k.clone()]
        bad[which][0, 1, at, 3] = value
        out, den2, _ = ops.normalized_fwd(bad[0], bad[1], v, 1e-5, False)
        den2, ref = den2.view(3, 448), den.view(3, 448)
        assert torch.equal(out[0, ::2], clean[0, ::2]) and torch.equal(den2[::2], ref[::2])  # other heads
        assert torch.equal(out[0, 1, :at], clean[0, 1, :at]) and torch.equal(den2[1, :at], ref[1, :at])
        assert not den2[1, at].isfinite()
        if which == 0:
            assert torch.equal(out[0, 1, at + 1:], clean[0, 1, at + 1:])
        else:
            assert not den2[1, at:].isfinite().any()
