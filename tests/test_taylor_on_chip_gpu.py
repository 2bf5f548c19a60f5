"""fla_taylor_attention_kernel (TaylorLinearAttention on raw q, k, the features formed on chip) against an
evaluation in 64 bits, at the edges of its chunks and of the shapes it takes."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _exact(q, k, v, g):
    q, k, v = (t.double().detach().requires_grad_(True) for t in (q, k, v))
    s = q @ k.transpose(-1, -2) / math.sqrt(q.shape[-1])
    out = torch.tril(1 + s + s * s / 2) @ v
    return (out.detach(),) + torch.autograd.grad(out, (q, k, v), g.double())


def _inputs(B, H, N, d, dv, bnhd=False):
    gen = torch.Generator(device=DEV).manual_seed(N + d + dv)

    def draw(width):
        shape = (B, N, H, width) if bnhd else (B, H, N, width)
        t = torch.randn(*shape, device=DEV, generator=gen).to(torch.bfloat16)
        return t.transpose(1, 2) if bnhd else t

    return draw(d), draw(d), draw(dv), draw(dv)


# one chunk, less than one, a ragged last one, one and many chunks of state; every value width
@pytest.mark.parametrize("B,H,N,d,dv,bnhd", [(1, 1, 32, 16, 64, False), (1, 2, 64, 8, 16, False), (2, 3, 128, 16, 32, True),
                                             (1, 2, 160, 16, 8, False), (1, 3, 192, 8, 64, True), (2, 2, 256, 16, 64, False),
                                             (1, 2, 1056, 16, 16, True), (1, 90, 320, 8, 32, False), (1, 2, 4160, 16, 64, False)])
def test_on_chip_features_against_64_bits(B, H, N, d, dv, bnhd):
    from flashy_linear_attention_b200 import TaylorLinearAttention, _lib, ops

    q, k, v, g = _inputs(B, H, N, d, dv, bnhd)
    tq, tk, tv = (t.detach().requires_grad_(True) for t in (q, k, v))
    out = TaylorLinearAttention.apply(tq, tk, tv)
    assert _lib.load().fla_sm100_last_launch_count() == 1
    grads = torch.autograd.grad(out, (tq, tk, tv), g)
    ops.check_status(torch.device(DEV))
    assert out.stride() == torch.empty_like(v).stride() and grads[2].stride() == torch.empty_like(v).stride()
    # Rounded to bf16 (2^-9 at most, 2^-9 / sqrt(3) in norm): the result, the features of both sides, the scores or
    # T, and the state: five roundings that add up in norm, each of the two kinds of terms having fewer
    for name, got, want in zip(("out", "dxq", "dxk", "dv"), (out,) + grads, _exact(q, k, v, g)):
        rel = ((got.double() - want).norm() / want.norm()).item()
        assert rel <= math.sqrt(5) * 2.0**-9 / math.sqrt(3) * 1.5, (name, rel)


def test_every_path_to_the_kernel_gives_the_same(monkeypatch):
    """The call prepared in Python instead of in the native host code; rows the kernel cannot read in place;
    gradients that are expanded. Values wider than 64 columns still go through features in memory."""
    from flashy_linear_attention_b200 import TaylorLinearAttention, _lib, ops

    q, k, v, g = _inputs(2, 3, 320, 16, 64)
    want = (ops.taylor_forward(q, k, v),) + tuple(ops.taylor_backward(g, q, k, v))
    odd = torch.zeros(2, 3, 320, 17, device=DEV, dtype=torch.bfloat16)
    odd[..., 1:] = q
    assert odd[..., 1:].data_ptr() % 16 != 0
    packed = (ops.taylor_forward(odd[..., 1:], k, v),) + tuple(ops.taylor_backward(g, odd[..., 1:], k, v))
    ones = torch.ones(1, 1, 1, 1, device=DEV, dtype=torch.bfloat16).expand(2, 3, 320, 64)
    spread = ops.taylor_backward(ones, q, k, v), ops.taylor_backward(ones.contiguous(), q, k, v)
    monkeypatch.setattr(_lib, "_host", False)
    plain = (ops.taylor_forward(q, k, v),) + tuple(ops.taylor_backward(g, q, k, v))
    for a, b, c in zip(want, packed, plain):
        assert torch.equal(a, b) and torch.equal(a, c)
    assert all(torch.equal(a, b) for a, b in zip(*spread))
    assert ops.taylor_forward(q, k, torch.cat([v, v], -1)) is None
    wide = TaylorLinearAttention.apply(q, k, torch.cat([v, v], -1))
    assert ((wide[..., :64].double() - want[0].double()).norm() / want[0].double().norm()).item() < 2.0**-7


# the narrowest and widest value widths on both sides of those that run on chip
@pytest.mark.parametrize("d", [8, 16])
@pytest.mark.parametrize("dv,kept", [(1, 2), (4, 2), (8, 0), (64, 0), (128, 2)])
def test_features_in_memory_are_formed_once(d, dv, kept):
    from flashy_linear_attention_b200 import TaylorLinearAttention

    q, k, v, g = _inputs(1, 3, 320, d, dv)
    tq, tk, tv = (t.requires_grad_(True) for t in (q, k, v))
    out = TaylorLinearAttention.apply(tq, tk, tv)
    assert len(out.grad_fn.saved_tensors) == 3 + kept
    grads = torch.autograd.grad(out, (tq, tk, tv), g)
    # as above, and with features in memory their gradients rounded too, each of which meets two terms
    for name, got, want in zip(("out", "dxq", "dxk", "dv"), (out,) + grads, _exact(q, k, v, g)):
        rel = ((got.double() - want).norm() / want.norm()).item()
        assert rel <= math.sqrt(7) * 2.0**-9 / math.sqrt(3) * 1.5, (name, rel)


# d = 8: both passes through memory; the forward alone; neither
@pytest.mark.parametrize("H,N,dv,bnhd,forward,kept", [(1, 4096, 64, True, False, 2), (3, 4160, 16, False, False, 2),
                                                      (16, 4096, 32, True, False, 0), (16, 3968, 32, False, True, 0)])
def test_few_long_heads_go_through_memory(H, N, dv, bnhd, forward, kept):
    from flashy_linear_attention_b200 import TaylorLinearAttention, ops

    q, k, v, g = _inputs(1, H, N, 8, dv, bnhd)
    assert (ops.taylor_forward(q, k, v) is not None) == forward
    tq, tk, tv = (t.detach().requires_grad_(True) for t in (q, k, v))
    out = TaylorLinearAttention.apply(tq, tk, tv)
    assert len(out.grad_fn.saved_tensors) == 3 + kept
    grads = torch.autograd.grad(out, (tq, tk, tv), g)
    ops.check_status(torch.device(DEV))
    assert out.stride() == torch.empty_like(v).stride() and grads[2].stride() == torch.empty_like(v).stride()
    for name, got, want in zip(("out", "dxq", "dxk", "dv"), (out,) + grads, _exact(q, k, v, g)):
        assert got.shape == want.shape
        rel = ((got.double() - want).norm() / want.norm()).item()
        assert rel <= math.sqrt(7) * 2.0**-9 / math.sqrt(3) * 1.5, (name, rel)


@pytest.mark.parametrize("d,dv", [(8, 64), (16, 128), (8, 4)])
def test_every_path_through_memory_gives_the_same(d, dv, monkeypatch):
    """The calls prepared in Python instead of in the native host code, rows of other strides or off a 16-byte
    boundary, an expanded gradient."""
    from flashy_linear_attention_b200 import _lib, ops

    def both(q, k, v, g):
        out, pq, pk = ops.taylor_forward_in_memory(q, k, v)
        return (out,) + tuple(ops.taylor_backward_in_memory(g, q, k, v, pq, pk))

    q, k, v, g = _inputs(2, 3, 320, d, dv)
    want = both(q, k, v, g)
    flat = torch.empty(q.numel() + 1, device=DEV, dtype=torch.bfloat16)
    off = flat[1:].view_as(q).copy_(q)
    assert off.is_contiguous() and off.data_ptr() % 16 != 0
    turned = k.transpose(1, 2).contiguous().transpose(1, 2)
    ones = torch.ones(1, 1, 1, 1, device=DEV, dtype=torch.bfloat16).expand(2, 3, 320, dv)
    other, spread = both(off, turned, v, g), both(q, k, v, ones)
    monkeypatch.setattr(_lib, "_host", False)
    for a, b in ((want, other), (want, both(q, k, v, g)), (want, both(off, turned, v, g)), (spread, both(q, k, v, ones.contiguous()))):
        assert all(torch.equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("dv", [24, 40, 72])
def test_value_widths_that_are_no_power_of_two_are_refused(dv):
    from flashy_linear_attention_b200 import TaylorLinearAttention

    q, k, v, _ = _inputs(1, 3, 320, 16, dv)
    with pytest.raises(AssertionError, match="power of 2"):
        TaylorLinearAttention.apply(q, k, v)


@pytest.mark.parametrize("backward", [False, True])
def test_a_tile_that_never_comes_ends_in_the_status_word(backward):
    from flashy_linear_attention_b200 import _lib, ops
    from flashy_linear_attention_b200._lib import FLA_DEBUG_WITHHOLD_FIRST_TILE, FlaArgs

    lib = _lib.load()
    q, k, v, g = _inputs(1, 2, 384, 16, 64)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = *q.shape, 64
    outs = [torch.empty_like(t) for t in (v, q, k, v)]
    for name, t in zip(("q", "k", "v", "d_o", "o", "d_q", "d_k", "d_v"), [q, k, v, g] + outs):
        setattr(a, name, ops._desc(t))
    a.stream = torch.cuda.current_stream(DEV).cuda_stream
    a.status, a.wait_limit_us, a.debug_flags = status.data_ptr(), 20000, FLA_DEBUG_WITHHOLD_FIRST_TILE
    call = lib.fla_sm100_taylor_bwd if backward else lib.fla_sm100_taylor_fwd
    assert call(ctypes.byref(a)) == 0
    torch.cuda.synchronize()
    assert int(status.item()) & 1
    recs = (ctypes.c_uint * (8 * 32))()
    assert lib.fla_sm100_timeout_records(recs, 32) >= 1
    # the same call without the hook
    status.zero_()
    a.debug_flags = 0
    assert call(ctypes.byref(a)) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    want = ops.taylor_backward(g, q, k, v) if backward else [ops.taylor_forward(q, k, v)]
    assert all(torch.equal(x, y) for x, y in zip(outs[1:] if backward else outs, want))


def test_shapes_the_c_entry_refuses():
    from flashy_linear_attention_b200 import _lib, ops
    from flashy_linear_attention_b200._lib import FlaArgs

    lib = _lib.load()
    q, k, v, _ = _inputs(1, 1, 128, 16, 64)
    for dk, dv, dtype in ((12, 64, 0), (16, 72, 0), (16, 64, 1)):
        a = FlaArgs()
        a.batch, a.heads, a.seqlen, a.dk, a.dv, a.dtype = 1, 1, 128, dk, dv, dtype
        a.q, a.k, a.v, a.o = ops._desc(q), ops._desc(k), ops._desc(v), ops._desc(torch.empty_like(v))
        assert lib.fla_sm100_taylor_fwd(ctypes.byref(a)) == -2
    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, 1, 128, 16, 64
    assert lib.fla_sm100_taylor_fwd(ctypes.byref(a)) == -1  # no tensors
