"""What autograd callers do around attention() beside a plain step, on the sorted and on the pairwise route."""

import pytest
import torch

from test_gpu_attention_sorted import KERNELS, PAIRWISE, SORTED, dense_attention, two_norm

pytestmark = pytest.mark.gpu


def inputs(D, S=100, B=2, H=2, C=16):
    g = torch.Generator().manual_seed(D)
    q, k, v = (torch.randn(B, H, S, n, generator=g).cuda().requires_grad_(True) for n in (D, D, C))
    return q, k, v, torch.randn(B, H, S, C, generator=g).cuda()


@pytest.mark.parametrize("D", [SORTED, PAIRWISE])
@pytest.mark.parametrize("kernel", KERNELS)
def test_output_changed_in_place(kernel, D):
    from kernel_attention import attention
    q, k, v, up = inputs(D)
    want = torch.autograd.grad(attention(q, k, v, kernel, 0.5), (q, k, v), 2 * up)
    out = attention(q, k, v, kernel, 0.5)
    out.mul_(2)
    out += q.detach()[..., :16]
    for a, b in zip(torch.autograd.grad(out, (q, k, v), up), want):
        assert two_norm(a, b) < 1e-5


def test_inputs_changed_in_place_are_refused():
    from kernel_attention import attention
    q, k, v, up = inputs(PAIRWISE)
    k2 = k * 1.0
    out = attention(q, k2, v, "add_laplace", 0.5)
    k2.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        out.backward(up)


def test_backward_twice_and_no_reference_cycle():
    import gc
    import weakref
    from kernel_attention import attention
    q, k, v, up = inputs(PAIRWISE)
    out = attention(q, k, v, "add_riesz", 0.5)
    first = torch.autograd.grad(out, (q, k, v), up, retain_graph=True)
    for a, b in zip(torch.autograd.grad(out, (q, k, v), up), first):
        assert torch.equal(a, b)
    gc.collect()
    gc.disable()
    try:
        out = attention(q, k, v, "add_riesz", 0.5)
        gone = weakref.ref(out)
        before = torch.cuda.memory_allocated()
        size = out.untyped_storage().nbytes()
        del out
        assert gone() is None and torch.cuda.memory_allocated() <= before - size
    finally:
        gc.enable()


@pytest.mark.parametrize("kernel", KERNELS)
def test_saved_tensor_hooks_that_hand_back_other_layouts(kernel):
    from kernel_attention import attention
    q, k, v, up = inputs(PAIRWISE)
    keep = (torch.arange(100, device="cuda")[None] < torch.tensor([[100], [60]], device="cuda"))
    want = torch.autograd.grad(attention(q, k, v, kernel, 0.5, keep), (q, k, v), up)

    def unpack(t):      # the same values, every other element of a new tensor, off its 16-byte boundary
        store = torch.full((2 * t.numel() + 1,), float("nan"), device="cuda")
        return store[1:].view(*t.shape[:-1], 2 * t.shape[-1])[..., ::2].copy_(t)

    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().cpu(), unpack):
        out = attention(q, k, v, kernel, 0.5, keep)
    out.mul_(1.0)
    for a, b in zip(torch.autograd.grad(out, (q, k, v), up), want):
        assert two_norm(a, b) < 1e-5
    from torch.utils.checkpoint import checkpoint
    out = checkpoint(lambda *x: attention(*x, kernel, 0.5, keep), q, k, v, use_reentrant=False)
    for a, b in zip(torch.autograd.grad(out, (q, k, v), up), want):
        assert two_norm(a, b) < 1e-5


@pytest.mark.parametrize("tau", ["per head", "trained", "negative", "one element"])
@pytest.mark.parametrize("kernel", KERNELS)
def test_temperatures(kernel, tau):
    from kernel_attention import attention
    q, k, v, up = inputs(PAIRWISE, S=60)
    tau = {"per head": torch.tensor([0.5, 0.8], device="cuda").view(1, 2, 1, 1), "trained": torch.tensor(0.7, device="cuda", requires_grad=True),
           "negative": -0.5, "one element": torch.tensor([0.6], device="cuda")}[tau]
    wrt = (q, k, v, tau) if isinstance(tau, torch.Tensor) and tau.requires_grad else (q, k, v)
    out, ref = attention(q, k, v, kernel, tau), dense_attention(q, k, v, kernel, tau, None)
    assert two_norm(out, ref) < 1e-5
    got, want = torch.autograd.grad(out, wrt, up), torch.autograd.grad(ref, wrt, up.double())
    for a, b in zip(got[:3], want[:3]):
        assert two_norm(a, b) < 2e-4
    if len(wrt) == 4:       # -(<grad_q, q> + <grad_k, k>) / tau, where the terms nearly cancel (add_riesz depends on tau through EPS only)
        bound = 2e-4 * sum((g.norm() * x.norm()).item() for g, x in zip(want[:2], (q, k))) / tau.item()
        assert (got[3] - want[3]).abs().item() < bound


@pytest.mark.parametrize("kernel", KERNELS)
def test_mask_that_wants_a_gradient(kernel):
    """A 0 / 1 mask of floats: kept keys get one, in the operators' sense."""
    from kernel_attention import attention
    q, k, v, up = inputs(PAIRWISE, S=60)
    keep = (torch.arange(60, device="cuda")[None] < torch.tensor([[60], [40]], device="cuda")).float().requires_grad_(True)
    out = attention(q, k, v, kernel, 0.5, keep)
    assert two_norm(out, dense_attention(q, k, v, kernel, 0.5, keep)) < 1e-5
    assert torch.autograd.grad(out, keep, up)[0].abs().max().item() > 0


def test_transforms_without_a_rule_are_refused():
    """Forward-mode derivatives, vmap and the functional transforms: an error, not a result without the derivative."""
    import torch.autograd.forward_ad as forward_ad
    from kernel_attention import attention
    from weighted_abs_sum import weighted_abs_sum, weighted_abs_sum_full
    from weighted_laplace_sum import weighted_laplace_sum
    g = torch.Generator(device="cuda").manual_seed(0)
    q, v, x = (torch.randn(*s, generator=g, device="cuda") for s in ((1, 2, 64), (1, 64, 4), (1, 2, 64, 4)))
    ops = [(f, (q, q + 1, v)) for f in (weighted_abs_sum, weighted_abs_sum_full, weighted_laplace_sum)]
    ops += [(lambda a, b, c, kernel=kernel: attention(a, b, c, kernel, 0.5), (x, x + 1, x)) for kernel in KERNELS]
    for f, args in ops:
        for grad_mode in (True, False):
            with torch.set_grad_enabled(grad_mode), forward_ad.dual_level(), pytest.raises(RuntimeError, match="jvp"):
                f(forward_ad.make_dual(args[0], torch.ones_like(args[0])), *args[1:])
        with pytest.raises(Exception):
            torch.func.vmap(f)(*(a[None] for a in args))
        with pytest.raises(Exception):
            torch.func.jvp(lambda a: f(a, *args[1:]), (args[0],), (args[0],))
        with pytest.raises(Exception):
            torch.func.grad(lambda a: sum(t.sum() for t in f(a, *args[1:])))(args[0])


@pytest.mark.filterwarnings("ignore")
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("name", ["abs", "abs_full", "laplace", *KERNELS])
def test_traced_calls_run_on_new_inputs(name, grad):
    from kernel_attention import attention
    from weighted_abs_sum import weighted_abs_sum, weighted_abs_sum_full
    from weighted_laplace_sum import weighted_laplace_sum
    call = {"abs": lambda q, k, v: weighted_abs_sum(q, k, v) * 2, "abs_full": lambda q, k, v: sum(t.sum(-1) if t.dim() == 3 else t for t in weighted_abs_sum_full(q, k, v)),
            "laplace": lambda q, k, v: weighted_laplace_sum(q, k, v)[0] * 2}.get(name, lambda q, k, v: attention(q, k, v, name, 0.5) * 2)
    g = torch.Generator(device="cuda").manual_seed(0)
    shapes = ((1, 2, 40, 8), (1, 2, 40, 8), (1, 2, 40, 4)) if name in KERNELS else ((2, 3, 40), (2, 3, 50), (2, 50, 4))
    first, second = ([torch.randn(*s, generator=g, device="cuda").requires_grad_(grad) for s in shapes] for _ in range(2))
    made = torch.jit.trace(call, tuple(first), check_trace=False)
    for compiled in (made, torch.compile(call, backend="aot_eager")):
        got, want = compiled(*second), call(*second)
        assert two_norm(got, want) < 1e-5
        if grad:
            for a, b in zip(torch.autograd.grad(got.sum(), second), torch.autograd.grad(want.sum(), second)):
                assert two_norm(a, b) < 1e-5
