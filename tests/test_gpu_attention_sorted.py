"""The sorted route of the attention entry points: layout change, masking, sums, normalisation and the gradients around the walks.
More features than the pairwise kernels take (128), so that no estimate of times decides which route runs; where a call must not
depend on the route, 16 features beside them, which run pair by pair at these lengths."""

import pytest
import torch

from util import rel_err

pytestmark = pytest.mark.gpu

KERNELS = ["add_laplace", "add_riesz", "add_bump"]
SORTED, PAIRWISE = 130, 16       # features


def dense_attention(q, k, v, kernel, tau, keep):
    """The attention by its definition in float64, differentiable; masked keys are left out."""
    q, k, v = q.double() / tau, k.double() / tau, v.double()
    x = (q[..., :, None, :] - k[..., None, :, :]).abs()
    if kernel == "add_laplace":
        A = torch.exp(-x).sum(-1)
    elif kernel == "add_bump":
        A = (1 - x).clamp_min(0).sum(-1)
    else:
        A = q.abs().sum(-1)[..., :, None] + k.abs().sum(-1)[..., None, :] - x.sum(-1) + 1e-3
    if keep is not None:
        A = A * keep[:, None, None, :].double()
    return (A @ v) / A.sum(-1, keepdim=True).clamp_min(1e-6)


def two_norm(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


def inputs(B, H, S, D, C, masked, seed):
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, H, S, n, generator=g).cuda() for n in (D, D, C))
    grad = torch.randn(B, H, S, C, generator=g).cuda()
    keep = None
    if masked:
        keep = (torch.rand(B, S, generator=g) > 0.4).cuda()
        keep[:, 0] = True
    return q, k, v, grad, keep


def call(q, k, v, grad, kernel, tau, keep, fn=None):
    """Output and gradients."""
    if fn is None:
        from kernel_attention import attention as fn
    q, k, v = (t.detach().clone().requires_grad_(True) for t in (q, k, v))
    out = fn(q, k, v, kernel, tau, keep)
    return (out.detach(), *torch.autograd.grad(out, (q, k, v), grad.to(out.dtype)))


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("B, H, S, C", [(1, 1, 1, 4), (2, 2, 64, 64), (1, 3, 129, 33), (2, 1, 300, 16), (1, 1, 700, 128), (3, 2, 90, 7)])
def test_outputs_and_gradients(B, H, S, C, kernel, masked):
    """Without autograd, with it, and its gradients, against the definition in float64."""
    from kernel_attention import attention
    q, k, v, grad, keep = inputs(B, H, S, SORTED, C, masked, S + C)
    if kernel == "add_bump":        # at least 1 / 64 from every kink: 23 million pairs of smooth values have some within rounding of one, each off by a whole slope
        q, k = (q * 64).round() / 64 + 1 / 128, (k * 64).round() / 64
    got = call(q, k, v, grad, kernel, 0.5, keep)
    want = call(q, k, v, grad, kernel, 0.5, keep, dense_attention)
    assert rel_err(attention(q, k, v, kernel, 0.5, keep), want[0]) < 1e-4
    assert rel_err(got[0], want[0]) < 1e-4
    for a, b in zip(got[1:], want[1:]):      # (one key: the gradients of q and k are rounding)
        assert two_norm(a, b) < 1e-4 or (S == 1 and (a.double() - b).abs().max().item() < 1e-6), two_norm(a, b)


@pytest.mark.parametrize("D", [SORTED, PAIRWISE])
@pytest.mark.parametrize("kernel", KERNELS)
def test_queries_at_zero_beside_masked_keys(kernel, D):
    """The sorted route moves masked keys to the origin: what they add where a query's coordinate is 0 (or, for the bump, one
    width from 0) has to be taken out with the derivative that the walk gave them there."""
    tau = 0.5
    q, k, v, grad, keep = inputs(2, 2, 150, D, 16, True, D)
    q[:, :, ::5, :7] = 0.0
    q[:, :, 3::5, 2:5] = -0.0
    q[:, :, 1::5, 3] = tau
    q[:, :, 2::5, 4] = -tau
    got = call(q, k, v, grad, kernel, tau, keep)
    want = call(q, k, v, grad, kernel, tau, keep, dense_attention)
    assert rel_err(got[0], want[0]) < 1e-4
    for a, b in zip(got[1:], want[1:]):
        assert two_norm(a, b) < 2e-4, two_norm(a, b)


@pytest.mark.parametrize("D", [SORTED, PAIRWISE])
@pytest.mark.parametrize("kernel", KERNELS)
def test_masked_values_are_never_looked_at(kernel, D):
    """Whatever stands in the masked rows of k and v, NaN and infinities too: the results are those of zeros there, and the masked
    rows get no gradient."""
    q, k, v, grad, keep = inputs(2, 2, 150, D, 16, True, 7 * D)
    junk = torch.tensor([float("nan"), float("inf"), -float("inf"), 3e38], device="cuda").repeat(38)[:150]
    off = ~keep[:, None, :, None]
    kj = torch.where(off, junk[:, None], k)
    vj = torch.where(off, junk[:, None].flip(0), v)
    got = call(q, kj, vj, grad, kernel, 0.5, keep)
    want = call(q, k.masked_fill(off, 0.0), v.masked_fill(off, 0.0), grad, kernel, 0.5, keep)
    for a, b in zip(got, want):      # (the same sums, in the order of the atomics)
        assert two_norm(a, b) < 1e-5, two_norm(a, b)
    for a in got[2:]:
        assert a.masked_select(off.expand_as(a)).abs().max().item() == 0.0
    from kernel_attention import attention
    assert two_norm(attention(q, kj, vj, kernel, 0.5, keep), want[0]) < 1e-5


@pytest.mark.parametrize("D", [SORTED, PAIRWISE])
@pytest.mark.parametrize("kernel", KERNELS)
def test_batch_without_any_key(kernel, D):
    """Every key of one batch entry masked: zeros come out there, no gradient goes in, and the other entry is not touched by it."""
    q, k, v, grad, keep = inputs(2, 2, 150, D, 16, True, 3 * D)
    keep[0] = False
    got = call(q, k, v, grad, kernel, 0.5, keep)
    alone = call(q[1:], k[1:], v[1:], grad[1:], kernel, 0.5, keep[1:])
    for a, b in zip(got, alone):
        assert a[0].abs().max().item() == 0.0
        assert two_norm(a[1:], b) < 1e-5
