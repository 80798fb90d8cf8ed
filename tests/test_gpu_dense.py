"""The pairwise kernels of short sequences at the edges of their tiles (64 rows, 16 or 32 features, 32 / 64 / 128 channels), with one CTA
and with a cluster per query tile, against the float64 definitions."""

import pytest
import torch

from oracle import direct
from util import make_inputs, rel_err

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1, 1), (2, 16, 63, 65, 32), (3, 17, 64, 64, 33), (1, 33, 65, 1, 64), (2, 128, 129, 200, 65), (1, 64, 700, 130, 128), (40, 15, 300, 257, 5)]


@pytest.mark.parametrize("shape", SHAPES)
def test_operators(shape):
    from weighted_abs_sum import weighted_abs_sum_full
    from weighted_laplace_sum import weighted_laplace_sum
    P, D, N, M, C = shape
    q, k, v = make_inputs(P, D, N, M, C, seed=N + M + D, scale=1.5)
    for got, want in ((weighted_laplace_sum(q, k, v), direct.laplace_sum(q, k, v)), (weighted_abs_sum_full(q, k, v), direct.abs_sum(q, k, v))):
        for a, b in zip(got, want):
            assert rel_err(a, b) < 2e-5, rel_err(a, b)


@pytest.mark.parametrize("kernel", ["add_laplace", "add_riesz", "add_bump"])
@pytest.mark.parametrize("shape", [(2, 2, 64, 16, 64), (1, 3, 129, 30, 33), (2, 1, 513, 128, 16), (3, 20, 190, 65, 100)])
def test_attention_masked(kernel, shape):
    """Scattered masks."""
    from kernel_attention import attention
    B, H, S, D, C = shape
    g = torch.Generator().manual_seed(S)
    q, k, v = torch.randn(B, H, S, D, generator=g), torch.randn(B, H, S, D, generator=g), torch.randn(B, H, S, C, generator=g)
    keep = torch.rand(B, S, generator=g) > 0.4
    keep[:, 0] = True
    out = attention(q.cuda(), k.cuda(), v.cuda(), kernel, 0.75, keep.cuda())
    want = direct.attention(q, k, v, kernel, 0.75, keep)
    assert rel_err(out, want) < 1e-4, rel_err(out, want)


@pytest.mark.parametrize("scale", [30.0, 200.0])
def test_laplace_values_beyond_the_exponential_range(scale):
    """Tiles with values above the range of e^x next to tiles without: both forms of a pair, mixed."""
    from weighted_laplace_sum import weighted_laplace_sum
    q, k, v = make_inputs(2, 5, 300, 200, 16, seed=4, ties=False)
    k[0, :, 70:100] *= scale
    k[1, 2, :] *= scale
    q[0, 1, 64:128] = k[0, 1, 64:128] + 0.5
    q[1, 2, :] = k[1, 2, :200] - 0.25
    for a, b in zip(weighted_laplace_sum(q, k, v), direct.laplace_sum(q, k, v)):
        assert torch.isfinite(a).all() and rel_err(a, b) < 2e-5, rel_err(a, b)


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("shape", [(1, 1, 1, 2, 1), (2, 16, 63, 65, 32), (3, 65, 64, 64, 33), (1, 128, 70, 129, 128), (2, 40, 400, 200, 5)])
def test_operator_gradients(shape, full):
    """With ties between queries and keys: the one-sided derivatives of the walk."""
    import qlka_native
    P, D, N, M, C = shape
    q, k, v = make_inputs(P, D, N, M, C, seed=N + M + D, scale=1.5)
    g = torch.Generator().manual_seed(7)
    g_w, g_u = torch.randn(P, M, C, generator=g).cuda(), torch.randn(P, M, generator=g).cuda() if full else None
    for got, want in ((qlka_native.laplace_backward(q, k, v, g_w, g_u), direct.laplace_sum_backward(q, k, v, g_w, g_u)),
                      (qlka_native.abs_backward(q, k, v, g_w, g_u), direct.abs_sum_backward(q, k, v, g_w, g_u))):
        for a, b in zip(got, want):
            assert rel_err(a, b) < 2e-5, rel_err(a, b)


def dense_attention(q, k, v, kernel, tau, keep):
    """The attention by its definition in float64, differentiable."""
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


@pytest.mark.parametrize("masked", [False, True])
@pytest.mark.parametrize("kernel", ["add_laplace", "add_riesz", "add_bump"])
@pytest.mark.parametrize("shape", [(2, 2, 64, 16, 64), (1, 3, 129, 30, 33), (2, 1, 300, 70, 16), (1, 1, 1500, 8, 64)])
def test_attention_gradients(kernel, shape, masked):
    """Forward and backward through autograd."""
    from kernel_attention import attention
    B, H, S, D, C = shape
    g = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(B, H, S, n, generator=g).cuda().requires_grad_(True) for n in (D, D, C))
    grad = torch.randn(B, H, S, C, generator=g).cuda()
    keep = None
    if masked:
        keep = (torch.rand(B, S, generator=g) > 0.4).cuda()
        keep[:, 0] = True
    out = attention(q, k, v, kernel, 0.5, keep)
    got = torch.autograd.grad(out, (q, k, v), grad)
    want_out = dense_attention(q, k, v, kernel, 0.5, keep)
    want = torch.autograd.grad(want_out, (q, k, v), grad.double())
    assert rel_err(out, want_out) < 1e-4
    for a, b in zip(got, want):     # (2-norm: a pair within rounding of a kink of the bump takes either slope)
        err = ((a.double() - b).norm() / b.norm()).item()
        assert err < 2e-4, err
