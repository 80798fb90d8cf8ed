"""Several host threads drive the library at once."""

import threading
import time

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["laplace", "abs", "attention"])
def test_a_call_that_waits_for_its_queue_keeps_no_other_thread(call):
    """A thread fills the queue of a stream that a kernel holds for about half a second, until its launches have to wait; this thread
    must keep running meanwhile."""
    from kernel_attention import attention
    from weighted_abs_sum import weighted_abs_sum_full
    from weighted_laplace_sum import weighted_laplace_sum
    q, v = torch.randn(1, 2, 64, device="cuda"), torch.randn(1, 64, 4, device="cuda")
    x = torch.randn(1, 1, 64, 4, device="cuda")
    run = {"laplace": lambda: weighted_laplace_sum(q, q, v), "abs": lambda: weighted_abs_sum_full(q, q, v),
           "attention": lambda: attention(x, x, x, "add_riesz", 1.0)}[call]
    run()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()

    def fill():
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)          # clocks: 0.5 s at the highest one
            for _ in range(3000):
                run()

    thread = threading.Thread(target=fill)
    thread.start()
    gap, last = 0.0, time.perf_counter()
    while thread.is_alive():
        time.sleep(0.001)
        now = time.perf_counter()
        gap, last = max(gap, now - last), now
    torch.cuda.synchronize()
    assert gap < 0.2, gap


def test_threads_on_their_own_streams_get_their_own_results():
    from kernel_attention import attention
    g = torch.Generator(device="cuda").manual_seed(0)
    inputs = [[torch.randn(2, 2, 300, n, generator=g, device="cuda").requires_grad_(True) for n in (16, 16, 8)] for _ in range(4)]

    def step(x):
        out = attention(*x, "add_laplace", 0.5)
        return (out.detach(), *torch.autograd.grad(out.sum(), x))

    want, got = [step(x) for x in inputs], [None] * 4
    torch.cuda.synchronize()

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                got[i] = step(inputs[i])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(got, want):
        for x, y in zip(a, b):
            assert ((x - y).norm() / y.norm()).item() < 1e-5
