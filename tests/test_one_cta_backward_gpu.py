"""fla_backward_kernel (the three gradients of a head in one CTA) against an evaluation in 64 bits: edges of its
chunks, head dims and dtypes, states before and after, and which calls take it."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture
def any_length():
    """Lifts the rule that the kernel only runs above 2048 tokens, so that short calls, which the 64-bit evaluation
    can follow, run in it."""
    from flashy_linear_attention_b200 import _lib, ops

    old = ops.set_debug_flags(_lib.FLA_DEBUG_FORCE_SINGLE_SWEEP)
    yield
    ops.set_debug_flags(old)


def _taken(heads, tokens, dim, flags=0):
    from flashy_linear_attention_b200 import _lib

    a = _lib.FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv, a.debug_flags = 1, heads, tokens, dim, dim, flags
    return _lib.load().fla_sm100_bwd_one_cta(ctypes.byref(a)) == 1


def _inputs(B, H, N, D, dtype, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    q, k = (torch.nn.functional.elu(torch.randn(B, H, N, D, device=DEV, generator=gen)) + 1 for _ in range(2))
    v, g = (torch.randn(B, H, N, D, device=DEV, generator=gen) for _ in range(2))
    if dtype == torch.float16:
        q = q / math.sqrt(D)
    return [t.to(dtype) for t in (q, k, v, g)]


def _exact(q, k, v, g, s0=None, r0=None):
    q, k, v, g = (t.double() for t in (q, k, v, g))
    p, dp = torch.tril(q @ k.mT), torch.tril(g @ v.mT)
    dq, dk, dv = dp @ k, dp.mT @ q, p.mT @ g
    if s0 is not None:
        dq = dq + g @ s0.double().mT
    if r0 is not None:
        dk, dv = dk + v @ r0.double().mT, dv + k @ r0.double()
    return dq, dk, dv, q.mT @ g + (0 if r0 is None else r0.double())


# every gradient rounds its two operands of each kind, scores or state, and the result: three roundings of
# 2^-9 (fp16: 2^-12) / sqrt(3) in norm; dq's and dk's score tiles have terms of both signs, which doubles theirs
def _bound(dtype):
    return (2.0**-9 if dtype == torch.bfloat16 else 2.0**-12) * math.sqrt((1 + 4 + 4) / 3)


def _run(q, k, v, g, s_last, **kw):
    from flashy_linear_attention_b200 import _lib, ops

    grads = ops.causal_dot_product_bwd(g, q, k, v, s_last=s_last, segments=1, **kw)
    assert _lib.load().fla_sm100_last_launch_count() == 1
    torch.cuda.synchronize()
    ops.check_status(torch.device(DEV))
    return grads


# ragged last chunks, the ring's second and third pass; 50 heads: the rule's edge below 64 columns, 99: from there
# on; 296 heads: two rounds
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,H,N,D", [(2, 50, 960, 128), (1, 99, 1024, 128), (4, 25, 1088, 83), (2, 64, 1344, 96), (1, 100, 1216, 128),
                                     (1, 50, 960, 56), (2, 32, 1024, 40), (1, 104, 1472, 64), (1, 99, 1216, 64), (2, 148, 448, 64)])
def test_gradients_against_64_bits(any_length, B, H, N, D, dtype):
    from flashlinear import LinearAttention
    from flashy_linear_attention_b200 import ops

    q, k, v, g = _inputs(B, H, N, D, dtype, N + D)
    assert ops.backward_uses_final_state(q, v) and _taken(B * H, N, D, ops._debug_flags)
    tq, tk, tv = (t.detach().requires_grad_(True) for t in (q, k, v))
    got = torch.autograd.grad(LinearAttention.apply(tq, tk, tv), (tq, tk, tv), g)
    ops.check_status(torch.device(DEV))
    for name, x, want in zip(("dq", "dk", "dv"), got, _exact(q, k, v, g)):
        rel = ((x.double() - want).norm() / want.norm()).item()
        assert rel <= _bound(dtype), (name, rel)


@pytest.mark.parametrize("with_s", [False, True])
@pytest.mark.parametrize("with_r", [False, True])
@pytest.mark.parametrize("H,N,D", [(100, 1024, 128), (100, 1096, 96), (100, 1024, 64), (64, 1100, 48)])
def test_states_before_and_after(any_length, H, N, D, with_s, with_r):
    assert _taken(H, N, D, 4)
    q, k, v, g = _inputs(1, H, N, D, torch.bfloat16, N)
    gen = torch.Generator(device=DEV).manual_seed(D)
    s0, r0 = (torch.randn(H, D, D, device=DEV, generator=gen) * 8 if w else None for w in (with_s, with_r))
    s_last = (k[0].double().mT @ v[0].double() + (s0.double() if with_s else 0)).float()
    r_final = torch.full((H, D, D), float("nan"), device=DEV)
    got = _run(q, k, v, g, s_last, s_init=s0, r_init=r0, r_final=r_final)
    want = _exact(q[0], k[0], v[0], g[0], s0, r0)
    for name, x, w in zip(("dq", "dk", "dv"), got, want):
        rel = ((x[0].double() - w).norm() / w.norm()).item()
        assert rel <= _bound(torch.bfloat16), (name, rel)
    # fp32 sums of N / 16 steps of 16 exact products
    assert ((r_final.double() - want[3]).norm() / want[3].norm()).item() <= (N / 16 + 2) * 2.0**-24


@pytest.mark.parametrize("with_s", [False, True])
@pytest.mark.parametrize("H,N,D", [(100, 1024, 128), (99, 1100, 64)])
def test_state_after_without_its_update(any_length, H, N, D, with_s):
    """r_init and no r_final: the R of the last chunk walked is never formed."""
    q, k, v, g = _inputs(1, H, N, D, torch.bfloat16, N)
    gen = torch.Generator(device=DEV).manual_seed(D)
    s0, r0 = (torch.randn(H, D, D, device=DEV, generator=gen) * 8 if w else None for w in (with_s, True))
    s_last = (k[0].double().mT @ v[0].double() + (s0.double() if with_s else 0)).float()
    got = _run(q, k, v, g, s_last, s_init=s0, r_init=r0)
    for name, x, w in zip(("dq", "dk", "dv"), got, _exact(q[0], k[0], v[0], g[0], s0, r0)):
        rel = ((x[0].double() - w).norm() / w.norm()).item()
        assert rel <= _bound(torch.bfloat16), (name, rel)


# one, two and three chunks: the first is the exact one, R is not formed, a state's copy is used once, a slot of the
# ring is filled a first and a second time; 445 heads: more than two rounds
@pytest.mark.parametrize("states", [False, True])
@pytest.mark.parametrize("H,N,D", [(99, 64, 128), (99, 128, 64), (100, 192, 128), (100, 250, 64), (99, 320, 96), (50, 384, 48),
                                   (445, 192, 128), (445, 320, 64)])
def test_few_chunks(any_length, H, N, D, states):
    q, k, v, g = _inputs(1, H, N, D, torch.bfloat16, N)
    gen = torch.Generator(device=DEV).manual_seed(D)
    s0, r0 = (torch.randn(H, D, D, device=DEV, generator=gen) * 8 if states else None for _ in range(2))
    s_last = (k[0].double().mT @ v[0].double() + (s0.double() if states else 0)).float()
    r_final = torch.full((H, D, D), float("nan"), device=DEV) if states else None
    got = _run(q, k, v, g, s_last, s_init=s0, r_init=r0, r_final=r_final)
    want = _exact(q[0], k[0], v[0], g[0], s0, r0)
    for name, x, w in zip(("dq", "dk", "dv"), got, want):
        rel = ((x[0].double() - w).norm() / w.norm()).item()
        assert rel <= _bound(torch.bfloat16), (name, rel)
    if states:  # fp32 sums of N / 16 steps of 16 exact products
        assert ((r_final.double() - want[3]).norm() / want[3].norm()).item() <= (N / 16 + 2) * 2.0**-24


def test_strided_inputs_and_guard_bands():
    """[B, H, N, D] views of [B, N, H, D] tensors; outputs' neighbours stay as they are."""
    from flashy_linear_attention_b200 import _lib, ops
    from flashy_linear_attention_b200._lib import FLA_DEBUG_FORCE_SINGLE_SWEEP, FlaArgs

    B, H, N, D = 1, 100, 1000, 128
    q, k, v, g = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in _inputs(B, H, N, D, torch.bfloat16, 3))
    s_last = (k[0].double().mT @ v[0].double()).float()
    frames = [torch.full((B, H, N + 4, D + 8), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    outs = [f[:, :, 2:N + 2, :D] for f in frames]
    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = B, H, N, D, D
    for name, t in zip(("q", "k", "v", "d_o", "d_q", "d_k", "d_v"), [q, k, v, g] + outs):
        setattr(a, name, ops._desc(t))
    a.s_last, a.debug_flags = s_last.data_ptr(), FLA_DEBUG_FORCE_SINGLE_SWEEP
    a.stream = torch.cuda.current_stream(DEV).cuda_stream
    lib = _lib.load()
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == 1
    assert lib.fla_sm100_bwd(ctypes.byref(a)) == 0
    torch.cuda.synchronize()
    for f, o, w in zip(frames, outs, _exact(q, k, v, g)):
        assert ((o.double() - w).norm() / w.norm()).item() <= _bound(torch.bfloat16)
        o.fill_(7.0)
        assert bool((f == 7.0).all())


@pytest.mark.parametrize("heads,dim,one", [(49, 56, 0), (50, 56, 1), (98, 64, 0), (99, 64, 1), (98, 128, 0), (99, 128, 1),
                                           (148, 128, 1), (149, 128, 0), (197, 128, 0), (198, 128, 1), (296, 128, 1)])
@pytest.mark.parametrize("tokens", [3136, 8192])
def test_calls_that_take_it_say_so(heads, dim, one, tokens):
    from flashy_linear_attention_b200 import _lib
    from flashy_linear_attention_b200._lib import FlaArgs

    a = FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, heads, tokens, dim, dim
    lib = _lib.load()
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == one and lib.fla_sm100_bwd_uses_final_state(ctypes.byref(a)) == 1
    a.dv = dim // 2
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == 0
    a.seqlen, a.dv = 2048, dim
    assert lib.fla_sm100_bwd_one_cta(ctypes.byref(a)) == 0 and lib.fla_sm100_bwd_uses_final_state(ctypes.byref(a)) == 0


@pytest.mark.parametrize("late", [float("inf"), float("nan"), 1000.0])
@pytest.mark.parametrize("H,N,D", [(99, 1024, 128), (128, 2048, 128), (128, 2048, 64)])
def test_no_later_token_reaches_dq_of_a_short_call(H, N, D, late):
    """dQ of a call of at most 2048 tokens is summed from the start: what the k and v of the last token hold
    changes no bit of the chunks before its own. The attention with its denominator likewise."""
    from flashlinear import LinearAttention
    from flashy_linear_attention_b200 import LinearAttentionNormalized

    q, k, v, g = _inputs(1, H, N, D, torch.bfloat16, 11)
    for function in (LinearAttention, LinearAttentionNormalized):
        dq = []
        for changed in (False, True):
            tq, tk, tv = (t.clone() for t in (q, k, v))
            if changed:
                tk[:, ::2, -1, 0] = late
                tv[:, 1::2, -1] *= late
            tq, tk, tv = (t.requires_grad_(True) for t in (tq, tk, tv))
            dq += torch.autograd.grad(function.apply(tq, tk, tv), tq, g)
        assert torch.equal(dq[0][:, :, :N - 128], dq[1][:, :, :N - 128])


@pytest.mark.parametrize("grow", [False, True], ids=["one large late row", "rows that grow"])
@pytest.mark.parametrize("H,N,D", [(99, 1024, 128), (99, 2176, 128), (99, 8192, 128), (99, 1920, 64), (99, 2304, 64)])
def test_dq_of_every_chunk_where_later_rows_are_larger(H, N, D, grow):
    """Chunk by chunk, as in a norm over all rows the large ones hide the rest. Above 2048 tokens the state before a
    chunk is the final state minus a sum over what follows: fp32 sums in steps of 16 tokens, each rounded by
    2^-24 of what it has grown to (at most the final state; the forward's and the backward's sum)."""
    from flashlinear import LinearAttention

    q, k, v, g = _inputs(1, H, N, D, torch.bfloat16, 12)
    if grow:
        v = (v.float() * torch.logspace(0, 3, N, device=DEV).view(1, 1, N, 1)).bfloat16()
    else:
        v[:, :, -1] *= 1000
    tq, tk, tv = (t.requires_grad_(True) for t in (q, k, v))
    got = torch.autograd.grad(LinearAttention.apply(tq, tk, tv), tq, g)[0]
    pick = slice(0, 3)
    q64, k64, v64, g64 = (t.detach()[:, pick].double() for t in (q, k, v, g))
    want = torch.tril(g64 @ v64.mT) @ k64
    total = (k64.mT @ v64).norm()
    for c in range(0, N, 128):
        rows = slice(c, c + 128)
        err = (got[:, pick, rows].double() - want[:, :, rows]).norm()
        sums = 2 * (N / 16 + 2) * 2.0**-24 * total * g64[:, :, rows].norm() if N > 2048 else 0.0
        # the same three roundings as above, of terms of both signs
        assert err <= _bound(torch.bfloat16) * want[:, :, rows].norm() + sums, c


def test_a_tile_that_never_comes_ends_in_the_status_word(any_length):
    from flashy_linear_attention_b200 import _lib, ops
    from flashy_linear_attention_b200._lib import FLA_DEBUG_FORCE_SINGLE_SWEEP, FLA_DEBUG_WITHHOLD_FIRST_TILE

    q, k, v, g = _inputs(1, 100, 1024, 128, torch.bfloat16, 5)
    s_last = (k[0].double().mT @ v[0].double()).float()
    want = _run(q, k, v, g, s_last)
    a = _lib.FlaArgs()
    a.batch, a.heads, a.seqlen, a.dk, a.dv = 1, 100, 1024, 128, 128
    outs = [torch.empty_like(t) for t in (q, k, v)]
    for name, t in zip(("q", "k", "v", "d_o", "d_q", "d_k", "d_v"), [q, k, v, g] + outs):
        setattr(a, name, ops._desc(t))
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    a.s_last, a.status, a.wait_limit_us = s_last.data_ptr(), status.data_ptr(), 20000
    a.stream = torch.cuda.current_stream(DEV).cuda_stream
    a.debug_flags = FLA_DEBUG_WITHHOLD_FIRST_TILE | FLA_DEBUG_FORCE_SINGLE_SWEEP
    lib = _lib.load()
    assert lib.fla_sm100_bwd(ctypes.byref(a)) == 0
    torch.cuda.synchronize()
    assert int(status.item()) & 1
    recs = (ctypes.c_uint * (8 * 32))()
    assert lib.fla_sm100_timeout_records(recs, 32) >= 1
    status.zero_()
    a.debug_flags = FLA_DEBUG_FORCE_SINGLE_SWEEP
    assert lib.fla_sm100_bwd(ctypes.byref(a)) == 0
    torch.cuda.synchronize()
    assert int(status.item()) == 0 and all(torch.equal(x, y) for x, y in zip(outs, want))
