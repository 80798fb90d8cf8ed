"""Gradients and the signed sum in pieces of their heads and features, as a smaller workspace or a nearly full device makes them go."""

import ctypes
import os
import subprocess
import sys

import pytest
import torch

from oracle import direct, sorted_scan
from util import rel_err

pytestmark = pytest.mark.gpu


def _inputs(P, D, N, M, C, device="cuda"):
    g = torch.Generator(device=device).manual_seed(P * N + M + C)
    r = lambda *s: torch.randn(*s, generator=g, device=device)
    return r(P, D, M), r(P, D, N), r(P, N, C), r(P, M, C), r(P, M)


def _tol(N, M):
    return 4 * (N + M + 128) * 2.0 ** -24          # as for the walks over events: roundings of 2^-24, no more than there are additions in a row


# heads that halve evenly and not, features that do and do not, channels that are padded; long segments with parts
@pytest.mark.parametrize("P,D,N,M,C", [(3, 130, 300, 200, 64), (5, 131, 70, 260, 33), (1, 133, 515, 513, 128), (2, 3, 17000, 20000, 16)])
def test_smaller_workspaces(P, D, N, M, C):
    import qlka_native
    lib = qlka_native.lib()
    q, k, v, g_w, g_u = _inputs(P, D, N, M, C)
    ref_l = direct.laplace_sum_backward(q, k, v, g_w, g_u) if N * M < 1 << 20 else sorted_scan.laplace_sum_backward(q, k, v, g_w, g_u)
    ref_a, ref_s = sorted_scan.abs_sum_backward(q, k, v, g_w, g_u), sorted_scan.sgn_sum(q, k, v, g_w)
    stream, dims = torch.cuda.current_stream().cuda_stream, (P, D, N, M, C)
    names = ("laplace_backward", "abs_backward", "sgn_forward")
    taken = {name: [] for name in names}
    for name in names:
        size = ctypes.c_size_t()
        assert getattr(lib, f"qlka_{name}_workspace_bytes")(*dims, ctypes.byref(size)) == 0
        for share in (1.0, 0.75, 0.5, 0.3, 0.15, 0.08, 0.02):
            have = int(size.value * share)
            ws = torch.empty(have, dtype=torch.uint8, device="cuda")
            out = [torch.full_like(x, float("nan")) for x in ((q,) if name == "sgn_forward" else (q, k, v))]
            if name == "sgn_forward":
                st = lib.qlka_weighted_sgn_sum_forward(q.data_ptr(), k.data_ptr(), v.data_ptr(), g_w.data_ptr(), out[0].data_ptr(), ws.data_ptr(), have, *dims, stream)
            else:
                st = getattr(lib, {"laplace_backward": "qlka_weighted_laplace_sum_backward", "abs_backward": "qlka_weighted_abs_sum_backward"}[name])(
                    q.data_ptr(), k.data_ptr(), v.data_ptr(), g_w.data_ptr(), g_u.data_ptr(), *[o.data_ptr() for o in out], ws.data_ptr(), have, *dims, stream)
            if st:
                assert st == 8, st                           # workspace too small
                continue
            taken[name].append(share)
            for a, b in zip(out, {"laplace_backward": ref_l, "abs_backward": ref_a, "sgn_forward": (ref_s,)}[name]):
                # (the roundings of the Laplace decays, which may all go the same way, have their own share: 2^-25 a key)
                assert rel_err(a, b) < _tol(N, M), (name, share, rel_err(a, b))
    for name in names:
        assert taken[name][0] == 1.0 and min(taken[name]) <= 0.5, taken


def test_device_that_is_nearly_full():
    """With three fifths of the workspace to be had, the results are the same; with a thirtieth, the allocator's error comes through. In a process of its
    own, whose allocator holds nothing else."""
    here = os.path.dirname(os.path.abspath(__file__))
    root = os.path.dirname(here)
    path = os.pathsep.join([here, root, os.path.join(root, "quasi-linear-kernel-attention_b200")])
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], env=dict(os.environ, PYTHONPATH=path), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def nearly_full(what):
    import qlka_native
    from kernel_attention.attention import attention
    P, D, N, C = 48, 64, 4096, 64
    size = ctypes.c_size_t()
    if what == "attention":
        q, k, v, g = (x.view(1, P, N, D).requires_grad_(i < 3) for i, x in enumerate(torch.randn(4, P, N, D, device="cuda", generator=torch.Generator("cuda").manual_seed(3))))
        assert qlka_native.lib().qlka_attention_backward_workspace_bytes(2, 1, P, N, D, C, 0, ctypes.byref(size)) == 0
        out = attention(q, k, v, "add_laplace", 0.5)
        call = lambda: torch.autograd.grad(out, (q, k, v), g, retain_graph=True)
    else:
        q, k, v, g_w, g_u = _inputs(P, D, N, N, C)
        assert getattr(qlka_native.lib(), f"qlka_{what}_backward_workspace_bytes")(P, D, N, N, C, ctypes.byref(size)) == 0
        call = lambda: getattr(qlka_native, f"{what}_backward")(q, k, v, g_w, g_u)
    want = [x.cpu() for x in call()]
    results = sum(x.numel() * 4 for x in want)

    def leave(free):             # this much beyond what the process holds now
        torch.cuda.empty_cache()
        total = torch.cuda.mem_get_info()[1]
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + free) / total)
        return torch.cuda.memory_stats()["num_ooms"]

    before = leave(results + int(0.6 * size.value))
    got = [x.cpu() for x in call()]
    assert torch.cuda.memory_stats()["num_ooms"] > before
    leave(results + size.value // 32)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        call()
    torch.cuda.set_per_process_memory_fraction(1.0)
    for a, b in zip(got, want):
        assert rel_err(a, b) < _tol(N, N)


if __name__ == "__main__":
    for case in ("laplace", "abs", "attention"):
        nearly_full(case)
