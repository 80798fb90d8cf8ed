"""The sort/rank stage on its own, through the C ABI: every array of the walk records
against a numpy restatement (bit-exact for the integer parts)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1, 1), (2, 3, 7, 5), (1, 2, 8, 9), (2, 2, 100, 77), (1, 3, 257, 300), (1, 2, 64, 1000),
          (1, 2, 1000, 3), (2, 2, 1024, 1024), (1, 2, 1025, 1500), (1, 2, 2049, 2048), (1, 2, 4096, 4000),
          (1, 2, 8191, 8192), (1, 2, 16384, 16384), (1, 1, 600, 16384)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("mode", [0, 1])
def test_records(shape, mode):
    P, D, N, M = shape
    g = torch.Generator().manual_seed(N * 7 + M)
    x = torch.randn(P, D, N, generator=g) * 3
    y = torch.randn(P, D, M, generator=g) * 3
    n = min(N, M, 4)
    x[0, 0, :n] = y[0, 0, :n]
    if N > 10:
        x[0, D - 1, 3:9] = x[0, D - 1, 2]
        x[0, 0, N // 2] = -0.0
        x[0, 0, N // 2 + 1] = 0.0
    check_records(x, y, mode)


# Key distributions that stress the sort and the rank search rather than the arithmetic: every key equal (one value bucket holds
# everything, and in the radix sort all lanes of a warp share every digit), two values, one far outlier (the bucket index of the rank search collapses to one bucket), keys already
# ascending / descending, values that differ only in their low mantissa bits, and infinities. Both the shared-memory kernel
# (N = 16384, 4096) and the long-sequence kernels (N = 20000).
KINDS = ["equal", "two_values", "outlier", "ascending", "descending", "low_bits", "infinities", "clump_40", "clump_200"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("N", [4096, 16384, 20000])
def test_records_degenerate_keys(kind, N):
    P, D, M = 1, 2, N - 37
    g = torch.Generator().manual_seed(N + len(kind))
    y = torch.randn(P, D, M, generator=g)
    if kind == "equal":
        x = torch.full((P, D, N), 0.75)
        y[0, 0, :100] = 0.75
    elif kind == "two_values":
        x = torch.where(torch.rand(P, D, N, generator=g) < 0.5, torch.tensor(-1.5), torch.tensor(0.25))
        y[0, 1, :50] = 0.25
    elif kind == "outlier":
        x = torch.randn(P, D, N, generator=g) * 0.01
        x[:, :, 17] = 3.0e6
        y = y * 0.01
    elif kind == "ascending":
        x = torch.linspace(-2.0, 2.0, N).repeat(P, D, 1).contiguous()
    elif kind == "descending":
        x = torch.linspace(2.0, -2.0, N).repeat(P, D, 1).contiguous()
    elif kind == "low_bits":
        x = (1.0 + torch.randint(0, 4096, (P, D, N), generator=g).float() * 2.0 ** -23)
        y = 1.0 + torch.randint(0, 4096, (P, D, M), generator=g).float() * 2.0 ** -23
    elif kind.startswith("clump"):
        # a group of equal keys inside smooth ones: 40 stay under the bucket sort's limit of 64 keys per bucket (ties are then
        # ranked inside the bucket), 200 send the segment to the radix sort
        x = torch.randn(P, D, N, generator=g)
        n = int(kind.split("_")[1])
        x[:, :, 100:100 + n] = 0.123
        y[0, 0, :30] = 0.123
    else:
        x = torch.randn(P, D, N, generator=g)
        x[:, :, 5] = float("inf")
        x[:, :, 9] = float("-inf")
    check_records(x, y, 1)
    if kind not in ("infinities", "outlier"):       # (Laplace weights of infinite or 1e6-wide gaps are 0 or NaN by definition; the ranks are what is tested here)
        check_records(x, y, 0)


@pytest.mark.parametrize("shape", [(1, 2, 20000, 17000), (1, 1, 40000, 300), (1, 1, 16385, 16385), (1, 1, 70001, 65536)])
@pytest.mark.parametrize("mode", [0, 1])
def test_records_long_segments(shape, mode):
    P, D, N, M = shape
    g = torch.Generator().manual_seed(N * 3 + M)
    x = torch.randn(P, D, N, generator=g) * 2
    y = torch.randn(P, D, M, generator=g) * 2
    x[0, 0, 3:9] = x[0, 0, 2]
    x[0, 0, :4] = y[0, 0, :4]
    check_records(x, y, mode)


# More queries than keys: parts are cut by their queries too, down to a few keys each, and a part whose queries crowd between two keys
# has more of them than a CTA holds.
@pytest.mark.parametrize("kind", ["plain", "narrow", "equal", "few_values", "one_key_value"])
@pytest.mark.parametrize("shape", [(1, 2, 1, 16385), (2, 1, 5, 40000), (1, 2, 300, 33000), (1, 1, 512, 70000), (1, 1, 2000, 262144), (1, 1, 8192, 100000), (1, 1, 20000, 30001)])
def test_records_more_queries_than_keys(shape, kind):
    P, D, N, M = shape
    g = torch.Generator().manual_seed(N + M)
    x, y = torch.randn(P, D, N, generator=g), torch.randn(P, D, M, generator=g)
    if kind == "narrow":
        y *= 0.01
    elif kind == "equal":
        y[:] = 0.3
        y[:, :, 7] = x[:, :, 0]
    elif kind == "few_values":
        x, y = (x * 2).round() / 2, (y * 2).round() / 2
    elif kind == "one_key_value":
        x[:] = 0.25
    for mode in (0, 1):
        check_records(x, y, mode)


# The list of events that the walks of the gradients read, and the marks at the keys where their first pass leaves checkpoints; above 16384
# keys or queries the segment is cut into parts, whose boundaries the blocks of 8 events do not respect.
@pytest.mark.parametrize("shape", [(1, 1, 1, 1), (2, 3, 7, 5), (1, 2, 8, 40), (1, 2, 257, 300), (1, 2, 1025, 1500), (1, 2, 64, 4000), (1, 2, 4000, 9), (1, 2, 16384, 16384),
                                   (2, 4, 20000, 20000), (1, 4, 65536, 65536), (1, 4, 40000, 8192), (1, 4, 8192, 40000), (2, 1, 5, 40000), (1, 1, 512, 70000), (1, 1, 2000, 262144)])
@pytest.mark.parametrize("kind", ["plain", "narrow", "few_values", "one_key_value"])
def test_events(shape, kind):
    P, D, N, M = shape
    g = torch.Generator().manual_seed(N * 5 + M)
    x, y = torch.randn(P, D, N, generator=g), torch.randn(P, D, M, generator=g)
    if kind == "narrow":             # queries crowd between few keys: more of them in a part than a CTA holds
        y *= 0.01
    elif kind == "few_values":
        x, y = (x * 2).round() / 2, (y * 2).round() / 2
    elif kind == "one_key_value":
        x[:] = 0.25
    for mode in (0, 1):
        check_events(x, y, mode)


def check_events(x, y, mode):
    import qlka_native
    P, D, N = x.shape
    M = y.shape[2]
    xperm, xval, eidx, esc, mstart = (t.cpu().numpy() for t in qlka_native.sort_rank_records(x.cuda(), y.cuda(), mode, events=True))
    _, _, yrec, want_ms = (t.cpu().numpy() for t in qlka_native.sort_rank_records(x.cuda(), y.cuda(), mode))      # (checked above)
    for s in range(P * D):
        xs, ys = x.numpy().reshape(P * D, N)[s], y.numpy().reshape(P * D, M)[s]
        word = xperm[s, :N].view(np.uint32)
        perm = (word & 0x3fffffff).astype(np.int64)
        sx = xs[perm]
        assert sorted(perm.tolist()) == list(range(N)) and np.all(sx[1:] >= sx[:-1])
        assert np.array_equal(mstart[s], want_ms[s])
        rank = np.sort(np.searchsorted(sx, ys, side="left"))                          # of the queries in walk order
        key_at, query_at = np.arange(N) + np.searchsorted(rank, np.arange(N), side="right"), np.arange(M) + rank
        e = eidx[s, :N + M].view(np.uint32)
        assert np.array_equal(e[key_at], perm.astype(np.uint32)), "a key's event"
        assert np.all(e[query_at] >> 31), "a query's event"
        rows = (e[query_at] & 0x7fffffff).astype(np.int64)
        assert sorted(rows.tolist()) == list(range(M))
        assert np.array_equal(np.searchsorted(sx, ys[rows], side="left"), rank), "queries not in rank order"
        # the queries' weights: those of their records, whichever of equal rank comes first
        by_row = np.empty((M, 2), np.int32)
        by_row[yrec[s, :M, 2]] = yrec[s, :M, :2]
        got = np.ascontiguousarray(esc[s, query_at]).view(np.int32)
        assert np.array_equal(got if mode == 0 else got[:, :1], by_row[rows] if mode == 0 else by_row[rows, :1])
        if mode == 1:
            assert np.array_equal(esc[s, key_at], np.stack([-2.0 * sx, np.zeros_like(sx)], 1))
            assert np.all(word >> 30 == 0)
            continue
        assert np.array_equal(esc[s, key_at], np.stack([xval[s, :N], np.zeros_like(sx)], 1))
        after = np.concatenate([[0], key_at[:-1] + 1])                                # the event right after the key before
        first = (np.arange(N) > 0) & (key_at // 8 != (after - 1) // 8)
        later = key_at // 8 != after // 8
        assert np.array_equal(word >> 31, first), f"{np.count_nonzero((word >> 31) != first)} marks of first keys"
        assert np.array_equal(word >> 30 & 1, later), f"{np.count_nonzero((word >> 30 & 1) != later)} marks of later keys"


def check_records(x, y, mode):
    import qlka_native
    P, D, N = x.shape
    M = y.shape[2]
    xperm, xval, yrec, mstart = (t.cpu().numpy() for t in qlka_native.sort_rank_records(x.cuda(), y.cuda(), mode))
    torch.cuda.synchronize()
    NBK = N // 8 + 1
    NP = NBK * 8
    xs_all, ys_all = x.numpy().reshape(P * D, N), y.numpy().reshape(P * D, M)
    for s in range(P * D):
        xs, ys = xs_all[s], ys_all[s]
        perm = xperm[s, :N].astype(np.int64)
        assert sorted(perm.tolist()) == list(range(N)), "xperm is not a permutation"
        sx = xs[perm]
        assert np.all(sx[1:] >= sx[:-1]), "keys not ascending"
        assert np.all(xperm[s, N:NP] == 0)
        if mode == 0:
            want = np.ones(NP + 8, np.float64)
            want[0] = 0.0
            want[1:N] = np.exp(-(sx[1:].astype(np.float64) - sx[:-1].astype(np.float64)))
            np.testing.assert_allclose(xval[s], want, rtol=2e-6, atol=1e-30)
        else:
            want = np.zeros(NP + 8, np.float32)
            want[:N] = sx
            assert np.array_equal(xval[s], want)
        assert yrec[s, M, 3] == -1, "sentinel record"
        rec = yrec[s, :M]
        rows = rec[:, 2].astype(np.int64)
        assert sorted(rows.tolist()) == list(range(M)), "query rows are not a permutation"
        sy = ys[rows]
        rank = rec[:, 3].astype(np.int64)
        assert np.all(rank[1:] >= rank[:-1]), "records not ordered by rank"       # equal ranks: any order
        assert np.array_equal(rank, np.searchsorted(sx, sy, side="left")), "rank != number of keys strictly below"
        e0, e1 = rec[:, 0].copy().view(np.float32), rec[:, 1].copy().view(np.float32)
        if mode == 0:
            w0 = np.where(rank > 0, np.exp(-(sy.astype(np.float64) - sx[np.maximum(rank - 1, 0)])), 0.0)
            w1 = np.where(rank < N, np.exp(-(sx[np.minimum(rank, N - 1)].astype(np.float64) - sy)), 0.0)
            # the query weights are taken with the hardware exponential: (2 + 1.2 gap) ulp
            g0 = np.where(rank > 0, sy.astype(np.float64) - sx[np.maximum(rank - 1, 0)], 0.0)
            g1 = np.where(rank < N, sx[np.minimum(rank, N - 1)].astype(np.float64) - sy, 0.0)
            assert np.all(np.abs(e0 - w0) <= (2e-6 + 1.5e-7 * g0) * w0 + 1e-37)
            assert np.all(np.abs(e1 - w1) <= (2e-6 + 1.5e-7 * g1) * w1 + 1e-37)
        else:
            assert np.array_equal(e0, 2.0 * sy)
        want_ms = np.concatenate([np.searchsorted(rank, np.arange(NBK) * 8, side="left"), [M]])
        assert np.array_equal(mstart[s, :NBK + 1].astype(np.int64), want_ms), "mstart"
