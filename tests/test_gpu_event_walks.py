"""The walks over events (dots, and rows and dots) and the first passes of all walks where their blocks, streams and channel groups begin and end."""

import pytest
import torch

from oracle import direct, sorted_scan
from util import rel_err

pytestmark = pytest.mark.gpu

D = 130        # more features than the pairwise kernels take: always the walks

# keys, queries, channels: lone events, blocks of 8 events full and not, streams of several warps, every lane layout with idle lanes and without
SIZES = [(1, 1, 1), (3, 5, 4), (8, 8, 33), (7, 10, 64), (16, 1, 40), (1, 41, 128), (130, 126, 32), (64, 300, 36), (515, 77, 100), (257, 1031, 64)]


def _inputs(N, M, C, where):
    g = torch.Generator().manual_seed(N * 7 + M * 3 + C)
    r = lambda *s: torch.randn(*s, generator=g)
    q, k = r(2, D, M), r(2, D, N)
    if where == "apart":             # all queries of a feature on one side of its keys, or crowded between two of them
        q[:, 0::3] = k[:, 0::3].amax(-1, keepdim=True) + 0.1 + q[:, 0::3].abs()
        q[:, 1::3] = k[:, 1::3].amin(-1, keepdim=True) - 0.1 - q[:, 1::3].abs()
        q[:, 2::3] = k[:, 2::3].mean(-1, keepdim=True) + 1e-3 * q[:, 2::3]
    return q, k, r(2, N, C), r(2, M, C), r(2, M)


def _tol(N, M):
    """Every result is a sum over keys (or queries) and channels in fp32: its rounding grows with the number of additions in a row, here no
    more than N + M + 128, each 2^-24 of sums that are at most a few times the largest result."""
    return 4 * (N + M + 128) * 2.0 ** -24


@pytest.mark.parametrize("where", ["mixed", "apart"])
@pytest.mark.parametrize("N,M,C", SIZES)
def test_laplace(N, M, C, where):
    import qlka_native
    q, k, v, g_w, g_u = _inputs(N, M, C, where)
    for gu in (g_u, None):
        got = qlka_native.laplace_backward(q.cuda(), k.cuda(), v.cuda(), g_w.cuda(), gu.cuda() if gu is not None else None)
        want = direct.laplace_sum_backward(q, k, v, g_w, gu if gu is not None else torch.zeros_like(g_u))
        for name, a, b in zip(("q", "k", "v"), got, want):
            assert rel_err(a, b) < _tol(N, M), (name, rel_err(a, b))


@pytest.mark.parametrize("where", ["mixed", "apart"])
@pytest.mark.parametrize("N,M,C", SIZES)
def test_abs_and_sgn(N, M, C, where):
    import qlka_native
    from weighted_abs_sum import weighted_sgn_sum
    q, k, v, g_w, g_u = _inputs(N, M, C, where)
    got = qlka_native.abs_backward(q.cuda(), k.cuda(), v.cuda(), g_w.cuda(), g_u.cuda())
    want = sorted_scan.abs_sum_backward(q, k, v, g_w, g_u)
    for name, a, b in zip(("q", "k", "v"), got, want):
        assert rel_err(a, b) < _tol(N, M), (name, rel_err(a, b))
    out, ref = weighted_sgn_sum(q.cuda(), k.cuda(), v.cuda(), g_w.cuda()), sorted_scan.sgn_sum(q, k, v, g_w)
    assert rel_err(out, ref) < _tol(N, M), rel_err(out, ref)


@pytest.mark.parametrize("where", ["mixed", "apart"])
@pytest.mark.parametrize("N,M,C", SIZES + [(1030, 515, 68), (2049, 2047, 8)])
def test_forward(N, M, C, where):
    import qlka_native
    q, k, v, _, _ = _inputs(N, M, C, where)
    for f, ref in ((qlka_native.laplace_forward, sorted_scan.laplace_sum), (lambda *x: qlka_native.abs_forward(*x, True), sorted_scan.abs_sum)):
        for a, b in zip(f(q.cuda(), k.cuda(), v.cuda()), ref(q, k, v)):
            assert rel_err(a, b) < _tol(N, M), rel_err(a, b)


# Above 16384 keys or queries a segment is cut by value into parts; 64 features, so that there are hundreds of part boundaries. Nearly equal
# lengths: the parts of the one order need more room than those of the longer side twice.
LONG = [(2, 64, 20000, 20000, 64), (1, 64, 65536, 65536, 32), (2, 64, 8192, 40000, 64), (2, 64, 40000, 8192, 64), (1, 64, 65535, 65536, 32), (2, 64, 16394, 16384, 64)]


def _long_inputs(P, D, N, M, C):
    g = torch.Generator().manual_seed(N + 3 * M)
    r = lambda *s: torch.randn(*s, generator=g)
    return r(P, D, M), r(P, D, N), r(P, N, C), r(P, M, C), r(P, M)


def _off(got, want, dim):
    """Largest relative error in the 2-norm over `dim` (a feature's whole gradient, or a row of grad_v's head)."""
    got, want = got.detach().double().cpu(), want
    return ((got - want).norm(dim=dim) / want.norm(dim=dim)).max().item()


def _long_tol(N, M, C):
    """Prefix sums: a state takes one rounded addition per key and a dot C more, twice N + M + C roundings of 2^-25 in the root mean square, which
    come together as their square root; products with keys, and sums whose terms cancel, are worth a factor of four."""
    return 4 * (2 * (N + M + C)) ** 0.5 * 2.0 ** -25


def _decay_tol(N, M):
    """Laplace: a step decay is rounded once, by 2^-25 at most and half of that on average, and these roundings need not cancel: between close keys
    the gaps are multiples of the keys' own spacing, so ties between two decays all go the same way. A state remembers
    keys about one unit back, 0.4 of all where N(0, 1) is densest. That bias (1.2e-4 at 20000) outgrows the rounding of the sums."""
    return 0.4 * max(N, M) * 2.0 ** -26


@pytest.mark.parametrize("with_u", [True, False])
@pytest.mark.parametrize("P,D_,N,M,C", LONG)
def test_long_laplace(P, D_, N, M, C, with_u):
    from weighted_laplace_sum import weighted_laplace_sum_backward
    q, k, v, g_w, g_u = _long_inputs(P, D_, N, M, C)
    g_u = g_u if with_u else None
    got = weighted_laplace_sum_backward(q.cuda(), k.cuda(), v.cuda(), g_w.cuda(), g_u.cuda() if with_u else None)
    want = sorted_scan.laplace_sum_backward(q, k, v, g_w, g_u)
    off = {name: _off(a, b, dim) for name, a, b, dim in zip(("q", "k", "v"), got, want, (-1, -1, 1))}
    assert max(off.values()) < _decay_tol(N, M), off


@pytest.mark.parametrize("with_u", [True, False])
@pytest.mark.parametrize("P,D_,N,M,C", LONG)
def test_long_abs_and_sgn(P, D_, N, M, C, with_u):
    from weighted_abs_sum import weighted_sgn_sum
    import qlka_native
    q, k, v, g_w, g_u = _long_inputs(P, D_, N, M, C)
    g_u = g_u if with_u else None
    got = qlka_native.abs_backward(q.cuda(), k.cuda(), v.cuda(), g_w.cuda(), g_u.cuda() if with_u else None)
    want = sorted_scan.abs_sum_backward(q, k, v, g_w, g_u)
    off = {name: _off(a, b, dim) for name, a, b, dim in zip(("q", "k", "v"), got, want, (-1, -1, 1))}
    if with_u:
        off["sgn"] = _off(weighted_sgn_sum(q.cuda(), k.cuda(), v.cuda(), g_w.cuda()), sorted_scan.sgn_sum(q, k, v, g_w), -1)
    assert max(off.values()) < _long_tol(N, M, C), off
