"""GPU tests of the native host path (csrc/fla_host.cpp) around what the kernels compute: other threads
and streams, and what autograd saves between forward and backward."""
import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _draw(*shape, seed=0, dtype=torch.bfloat16):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(*shape, device=DEV, generator=gen).to(dtype)


def test_other_threads_run_while_a_call_blocks():
    """Calls behind a long kernel fill the launch queue and block; the interpreter stays free."""
    from flashy_linear_attention_b200 import ops

    q = _draw(1, 2, 128, 64)
    ops.causal_dot_product_fwd(q, q, q)
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.002)

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(1_500_000_000)  # three quarters of a second
        t0 = time.perf_counter()
        for _ in range(3000):
            ops.host_forward(q, q, q)
        blocked = time.perf_counter() - t0
        torch.cuda.synchronize()
    finally:
        stop.set()
        thread.join()
    gaps = [b - a for a, b in zip(ticks, ticks[1:])]
    assert blocked > 0.3, "the launch queue never filled: the test shows nothing"
    assert max(gaps) < 0.2, max(gaps)


@pytest.mark.parametrize("shape", [(2, 3, 192, 83), (1, 2, 2240, 64), (1, 4, 4096, 128), (1, 2, 128, 192)],
                         ids=lambda s: "x".join(map(str, s)))
def test_calls_without_the_native_host_path_give_the_same(shape, monkeypatch):
    """Same kernels, same plan (final state and boundary states included), other host code."""
    from flashy_linear_attention_b200 import LinearAttention, _lib

    q, k, v, g = (_draw(*shape, seed=i) for i in range(4))

    def step():
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        out = LinearAttention.apply(*x)
        return (out,) + torch.autograd.grad(out, x, g)

    want = step()
    monkeypatch.setattr(_lib, "_host", False)
    for a, b in zip(step(), want):
        assert torch.equal(a, b) and a.stride() == b.stride()


def _odd(layout, B=2, H=3, N=192, d=83, seed=0):
    x = _draw(B, N, H, d, seed=seed).transpose(1, 2)
    return x if layout == "bnhd" else x.contiguous()


def _step(x, g):
    from flashy_linear_attention_b200 import LinearAttention

    out = LinearAttention.apply(*x)
    return (out,) + torch.autograd.grad(out, x, g)


@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
def test_a_layer_holds_one_copy_of_an_odd_head_dim(layout):
    """Between forward and backward an odd head dim costs what its repacked rows take (88 columns for 83), not
    that and q, k, v as well, and the gradients have the layout of q, k, v."""
    from flashy_linear_attention_b200 import LinearAttention

    leaf = [_odd(layout, N=2048, seed=i).requires_grad_(True) for i in range(3)]
    g = _odd(layout, N=2048, seed=3)
    _step(leaf, g)
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    out = LinearAttention.apply(*(t * 1 for t in leaf))  # nobody else keeps the three products
    torch.cuda.synchronize()
    rows = leaf[0].numel() // 83
    held = torch.cuda.memory_allocated() - before - rows * 83 * 2  # without the output
    assert held < 1.1 * 3 * rows * 88 * 2, held / (3 * rows * 88 * 2)
    x = [t.detach().requires_grad_(True) for t in leaf]
    for got, want, t in zip(torch.autograd.grad(out, leaf, g), _step(x, g)[1:], leaf):
        assert torch.equal(got, want) and want.stride() == torch.empty_like(t).stride()


@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("d", [83, 64])
def test_an_input_changed_in_place_before_the_backward_is_refused(which, d):
    from flashy_linear_attention_b200 import LinearAttention

    leaf = [_odd("bhnd", d=d, seed=i).requires_grad_(True) for i in range(3)]
    x = [t * 1 for t in leaf]
    out = LinearAttention.apply(*x)
    with torch.no_grad():
        x[which].add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out.sum(), leaf)


@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
@pytest.mark.parametrize("d", [83, 64])
def test_saved_tensors_may_come_back_elsewhere_and_contiguous(layout, d):
    """saved_tensors_hooks that move what is saved to the host and bring back plain contiguous tensors."""
    x = [_odd(layout, N=2240, d=d, seed=i).requires_grad_(True) for i in range(3)]
    g = _odd(layout, N=2240, d=d, seed=3)
    want = _step(x, g)
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu().contiguous(), lambda t: t.to(DEV)):
        got = _step(x, g)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    with torch.autograd.graph.save_on_cpu():
        got = _step(x, g)
    for a, b in zip(got, want):
        assert torch.equal(a, b) and a.stride() == b.stride()


@pytest.mark.parametrize("d", [83, 64])
def test_two_threads_on_streams_of_their_own(d):
    """Each thread's forward and backward on its own stream, inputs made there; many at once."""
    results, errors = {}, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for rep in range(20):
                    x = [_odd("bhnd", N=512, d=d, seed=10 * i + j).requires_grad_(True) for j in range(3)]
                    got = [t.clone() for t in _step(x, _odd("bhnd", N=512, d=d, seed=10 * i + 9))]
                    first = results.setdefault(i, got)
                    torch.cuda.current_stream().synchronize()
                    assert all(torch.equal(a, b) for a, b in zip(first, got)), (i, rep)
        except Exception as exc:  # reported by the main thread
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    torch.cuda.synchronize()
    for i, got in results.items():
        x = [_odd("bhnd", N=512, d=d, seed=10 * i + j).requires_grad_(True) for j in range(3)]
        for a, b in zip(got, _step(x, _odd("bhnd", N=512, d=d, seed=10 * i + 9))):
            assert torch.equal(a, b)


def test_gradients_of_repacked_inputs_take_the_layout_of_empty_like():
    """Permuted, expanded and sliced inputs whose rows have to be repacked."""
    from flashy_linear_attention_b200 import LinearAttention

    base = _draw(2, 3, 128, 90, seed=1)
    forms = [base[..., :83].contiguous(), base[..., :83], base[..., 1:84], base[:, :, :, :83].transpose(1, 2).contiguous().transpose(1, 2),
             base[..., :83].transpose(0, 1).contiguous().transpose(0, 1), base[:, :1, :, :83].expand(2, 3, 128, 83),
             base[..., :83].transpose(2, 3).contiguous().transpose(2, 3), base[:1, ..., :83].contiguous().expand(2, 3, 128, 83)]
    g = _draw(2, 3, 128, 83, seed=2)
    for i, x in enumerate(forms):
        leaf = [x.detach().requires_grad_(True)] + [forms[0].detach().clone().requires_grad_(True) for _ in range(2)]
        got = torch.autograd.grad(LinearAttention.apply(*leaf), leaf, g)
        plain = [t.detach().contiguous().requires_grad_(True) for t in leaf]
        want = torch.autograd.grad(LinearAttention.apply(*plain), plain, g)
        for a, b, t in zip(got, want, leaf):
            assert torch.equal(a, b) and a.stride() == torch.empty_like(t).stride(), (i, a.stride(), t.stride())
