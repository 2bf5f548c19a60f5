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
