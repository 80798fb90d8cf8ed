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
