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
    """Padded and scattered masks; a masked key counts nothing even if its values are not finite."""
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
