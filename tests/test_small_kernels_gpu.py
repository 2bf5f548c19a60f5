"""GPU tests of the small kernels beside the attention kernels: the recurrent kernel that takes
forward calls of a few tokens, and the row pad / unpad kernels."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens: one, an odd few, the longest calls of the recurrent kernel (16, for head dims up to 64: 8)
# and the shortest beyond them;
# head dims: a whole tile, columns that are no multiple of 4 or of a block's 32, one block, dk != dv
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [1, 3, 4, 5, 8, 9, 16, 17])
@pytest.mark.parametrize("dk,dv", [(128, 128), (83, 83), (64, 40), (8, 128), (128, 8)])
def test_few_tokens_from_a_state(tokens, dk, dv, dtype):
    from flashy_linear_attention_b200 import LinearAttentionResumable

    gen = torch.Generator(device="cuda").manual_seed(tokens * 1000 + dk + dv)
    B, H = 2, 3
    q, k = (torch.randn(B, tokens, H, dk, device="cuda", generator=gen).to(dtype).transpose(1, 2) / dk**0.5
            for _ in range(2))
    v = torch.randn(B, H, tokens, dv, device="cuda", generator=gen).to(dtype)
    s0 = torch.randn(B, H, dk, dv, device="cuda", generator=gen)
    for state in (s0, None):
        out, s1 = LinearAttentionResumable.apply(q, k, v, state)
        qd, kd, vd = q.double(), k.double(), v.double()
        start = torch.zeros_like(s0).double() if state is None else s0.double()
        want = qd @ start + torch.tril(qd @ kd.transpose(-1, -2)) @ vd
        want_s = start + kd.transpose(-1, -2) @ vd
        # fp32 sums of at most tokens + 1 terms of size <= max|s|
        assert (s1.double() - want_s).abs().max() <= 2e-6 * (tokens + 1) * want_s.abs().max()
        # one rounding of the result (half an ulp: 2^-9 / 2^-12 relative); beyond that the state
        # and the scores are rounded to 16 bits as well, three roundings that add up in norm
        ulp = 2.0**-9 if dtype == torch.bfloat16 else 2.0**-12
        rounds = 1 if tokens <= (16 if max(dk, dv) > 64 else 8) else 3
        rel = (out.double() - want).norm() / want.norm()
        assert rel <= rounds * ulp, (rel.item(), rounds * ulp)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [1, 2, 5, 8, 16])
def test_few_tokens_round_the_state_once(tokens, dtype):
    """A running state much larger than what a call adds to it, as after a few hundred tokens: the new one
    is the exact sum rounded to fp32 once. The sum of the call's own tokens, itself in fp32, is off by at most
    tokens x 2^-24 of its size, which is 1 / 16 or less of the state's here: a tenth of the rounding in norm."""
    from flashy_linear_attention_b200 import LinearAttentionResumable

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    B, H, d = 2, 8, 128
    q, k, v = (torch.randn(B, H, tokens, d, device="cuda", generator=gen).to(dtype) for _ in range(3))
    s0 = torch.randn(B, H, d, d, device="cuda", generator=gen) * 64
    _, s1 = LinearAttentionResumable.apply(q, k, v, s0)
    want = s0.double() + k.double().transpose(-1, -2) @ v.double()
    once = (want.float().double() - want).norm()
    assert (s1.double() - want).norm() <= 1.1 * once


@pytest.mark.parametrize("tokens", [4, 7, 16])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_few_tokens_keep_what_comes_before_a_bad_one(tokens, value):
    from flashy_linear_attention_b200 import LinearAttentionResumable

    gen = torch.Generator(device="cuda").manual_seed(tokens)
    q, k, v = (torch.randn(1, 3, tokens, 128, device="cuda", generator=gen).bfloat16() for _ in range(3))
    s0 = torch.randn(1, 3, 128, 128, device="cuda", generator=gen)
    clean, state = LinearAttentionResumable.apply(q, k, v, s0)
    at = tokens - 2
    for which in range(3):
        x = [q.clone(), k.clone(), v.clone()]
        x[which][0, 1, at, 5] = value
        out, s1 = LinearAttentionResumable.apply(*x, s0)
        assert torch.equal(out[0, ::2], clean[0, ::2]) and torch.equal(s1[0, ::2], state[0, ::2])
        assert torch.equal(out[0, 1, :at], clean[0, 1, :at]) and not out[0, 1, at].isfinite().all()
        if which == 0:  # a query leaves no trace
            assert torch.equal(out[0, 1, at + 1:], clean[0, 1, at + 1:]) and torch.equal(s1, state)
        else:
            assert not out[0, 1, at + 1].isfinite().all() and not s1[0, 1].isfinite().all()


# one token whose row is no multiple of 16 bytes although its head and batch strides are or do not
# count: a tensor of its own, one step of a longer contiguous one (at a 16-byte boundary and not)
@pytest.mark.parametrize("d", [83, 20])
@pytest.mark.parametrize("step", [None, 0, 8, 3])
def test_one_token_with_an_odd_row(d, step):
    from flashy_linear_attention_b200 import LinearAttentionResumable, ops

    gen = torch.Generator(device="cuda").manual_seed(d)
    H = 1 if step is None else 3

    def draw():
        n = 1 if step is None else 64
        t = torch.randn(1, H, n, d, device="cuda", generator=gen).bfloat16()
        return t if step is None else t[:, :, step:step + 1]

    q, k, v, g = (draw() for _ in range(4))
    s0 = torch.randn(1, H, d, d, device="cuda", generator=gen)
    out, s1 = LinearAttentionResumable.apply(q, k, v, s0)
    want_s = s0.double() + k.double().transpose(-1, -2) @ v.double()
    want = q.double() @ want_s
    assert (s1.double() - want_s).abs().max() <= 4e-6 * want_s.abs().max()
    assert (out.double() - want).norm() <= 2.0**-9 * want.norm()  # one rounding of the result
    general = ops.causal_dot_product_fwd(q, k, v, s_init=s0.view(H, d, d), s_final=torch.empty(H, d, d, device="cuda"))
    assert torch.equal(out, general)  # the Python path judges the strides like the native one
    dq, dk, dv = ops.causal_dot_product_bwd(g, q, k, v)
    p, dp = (q.double() * k.double()).sum(-1, keepdim=True), (g.double() * v.double()).sum(-1, keepdim=True)
    for got, ref in ((dq, dp * k.double()), (dk, dp * q.double()), (dv, p * g.double())):
        assert (got.double() - ref).norm() <= 1e-2 * ref.norm()


def test_few_tokens_state_in_place():
    from flashy_linear_attention_b200 import ops

    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(1, 4, 3, 128, device="cuda", generator=gen).bfloat16() for _ in range(3))
    state = torch.randn(4, 128, 128, device="cuda", generator=gen)
    other = torch.empty_like(state)
    out = ops.causal_dot_product_fwd(q, k, v, s_init=state, s_final=other)
    out2 = ops.causal_dot_product_fwd(q, k, v, s_init=state, s_final=state)
    assert torch.equal(out, out2) and torch.equal(state, other)


# rows of one element, pieces that cross one row end, several, none; a last block with few rows;
# destinations that are 16-byte aligned and only 4-byte aligned
@pytest.mark.parametrize("rows", [1, 31, 33, 1000])
@pytest.mark.parametrize("d", [1, 3, 7, 9, 16, 83, 273])
@pytest.mark.parametrize("offset", [0, 2])
def test_pad_and_unpad_rows_batch(rows, d, offset):
    from flashy_linear_attention_b200 import _lib

    lib = _lib.load()
    dpad = (d + 7) // 8 * 8
    n = 3
    src = [torch.randn(rows * d + 8, device="cuda").bfloat16()[offset:offset + rows * d] for _ in range(n)]
    mid = [torch.full((rows, dpad), 7.0, device="cuda").bfloat16() for _ in range(n)]
    buf = [torch.full((rows * d + 64,), 5.0, device="cuda").bfloat16() for _ in range(n)]
    dst = [b[8 + offset:8 + offset + rows * d] for b in buf]
    stream = torch.cuda.current_stream().cuda_stream
    arr = lambda ts: (ctypes.c_void_p * n)(*[t.data_ptr() for t in ts])  # noqa: E731
    assert lib.fla_sm100_pad_rows_batch(arr(src), arr(mid), n, rows, d, dpad, stream) == 0
    assert lib.fla_sm100_unpad_rows_batch(arr(mid), arr(dst), n, rows, d, dpad, stream) == 0
    for s, m, t, b in zip(src, mid, dst, buf):
        assert torch.equal(m[:, :d], s.view(rows, d)) and not m[:, d:].any()
        assert torch.equal(t, s)
        assert (b[:8 + offset] == 5).all() and (b[8 + offset + rows * d:] == 5).all()  # nothing beyond


# head dims that are no multiple of 8: odd and even ones, one column, one column into the second
# 64-column group, one short of a tile; lengths with whole and partly used chunks
@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,dk,dv", [(64, 83, 83), (320, 63, 63), (192, 1, 1), (256, 65, 65), (352, 127, 127),
                                     (2240, 90, 90), (192, 20, 64), (160, 64, 20), (200, 83, 83)])
def test_head_dims_that_are_no_multiple_of_8(N, dk, dv, dtype, layout):
    from flashy_linear_attention_b200 import LinearAttentionResumable, ops

    gen = torch.Generator(device="cuda").manual_seed(N + dk)
    B, H = 2, 3

    def draw(d, scale=1.0):
        x = (torch.randn(B, N, H, d, device="cuda", generator=gen) * scale).to(dtype).transpose(1, 2)
        return x if layout == "bnhd" else x.contiguous()

    q, k, v, g = draw(dk, dk**-0.5), draw(dk), draw(dv), draw(dv)
    out, s_final, seg_states, views = ops.host_forward(q, k, v, None, 2)
    grads = ops.host_backward(g, q, k, v, s_last=s_final, seg_states=seg_states, views=views)[:3]
    plain = ops.host_backward(g, q, k, v, s_last=s_final, seg_states=seg_states)[:3]
    for a, b, t in zip(grads, plain, (q, k, v)):
        assert torch.equal(a, b) and a.stride() == torch.empty_like(t).stride()
    assert out.stride() == torch.empty_like(v).stride()
    qd, kd, vd, gd = (t.double() for t in (q, k, v, g))
    P, dP = torch.tril(qd @ kd.transpose(-1, -2)), torch.tril(gd @ vd.transpose(-1, -2))
    want = (P @ vd, dP @ kd, dP.transpose(-1, -2) @ qd, P.transpose(-1, -2) @ gd)
    # scores, state and result rounded to 16 bits: three roundings of half an ulp, and room for the
    # cancellation of the total-minus-suffix form at 2240 tokens
    bound = 1e-2 if dtype == torch.bfloat16 else 2e-3
    for got, ref in zip((out,) + tuple(grads), want):
        assert (got.double() - ref).norm() / ref.norm() < bound
    if N % 32 == 0:
        o2, s2 = LinearAttentionResumable.apply(q, k, v)
        assert torch.equal(o2, ops.causal_dot_product_fwd(q, k, v)) and s2.shape == (B, H, dk, dv)
