"""Walk emission at its edges: both lane mappings of the row walks at every row width, blocks with none, some and more queries than
a slot stages (rounded values put many queries before one key), against the float64 definitions. More features than the pairwise
kernels take, so that the walks run."""

import pytest
import torch

from oracle import direct
from util import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid", [None, 0.5])
@pytest.mark.parametrize("N,M", [(1, 1), (9, 200), (64, 16), (64, 17), (64, 64), (65, 66), (300, 65), (1000, 1000)])
@pytest.mark.parametrize("C", [4, 32, 33, 64, 65, 128])
def test_walk_emission(C, N, M, grid):
    from weighted_abs_sum import weighted_abs_sum_full, weighted_sgn_sum
    from weighted_laplace_sum import weighted_laplace_sum, weighted_laplace_sum_backward
    P, D = 2, 130
    gen = torch.Generator(device="cuda").manual_seed(N + M + C)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    q, k, v, g_w, g_u = rnd(P, D, M), rnd(P, D, N), rnd(P, N, C), rnd(P, M, C), rnd(P, M)
    if grid:
        q, k = (q / grid).round() * grid, (k / grid).round() * grid
    out_w, out_u = weighted_laplace_sum(q, k, v)
    ref_w, ref_u = direct.laplace_sum(q, k, v)
    assert rel_err(out_w, ref_w) < 1e-4 and rel_err(out_u, ref_u) < 1e-4
    for got, want in zip(weighted_laplace_sum_backward(q, k, v, g_w, g_u), direct.laplace_sum_backward(q, k, v, g_w, g_u)):
        assert rel_err(got, want) < 1e-4
    out_w, out_u = weighted_abs_sum_full(q, k, v)
    ref_w, ref_u = direct.abs_sum(q, k, v)
    assert rel_err(out_w, ref_w) < 1e-4 and rel_err(out_u, ref_u) < 1e-4
    assert rel_err(weighted_sgn_sum(q, k, v, g_w), direct.sgn_sum(q, k, v, g_w)) < 1e-4


@pytest.mark.parametrize("full", [False, True])
@pytest.mark.parametrize("N,M", [(9, 200), (64, 17), (65, 66), (300, 65), (1000, 1000)])
@pytest.mark.parametrize("C", [4, 33, 64, 65, 128])
def test_walk_emission_abs_gradients(C, N, M, full):
    """grad_q by dots, grad_k and grad_v from one walk, at every row width; values on a grid put many queries before one key."""
    from qlka_native import abs_backward
    P, D = 2, 130
    gen = torch.Generator(device="cuda").manual_seed(N + M + C)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    q, k, v, g_w = (rnd(P, D, M) * 2).round() / 2, rnd(P, D, N), rnd(P, N, C), rnd(P, M, C)
    k[:, ::2] = (k[:, ::2] * 2).round() / 2
    g_u = rnd(P, M) if full else None
    for got, want in zip(abs_backward(q, k, v, g_w, g_u), direct.abs_sum_backward(q, k, v, g_w, g_u)):
        assert rel_err(got, want) < 1e-4
