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
                                   (1, 2, 256, 8), (1, 130, 2176, 64)], ids=lambda s: "x".join(map(str, s)))
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
