"""The encoder's linear layers on the bf16 tensor cores: at most the error of torch's fp32 product against float64, at the edges
of the 128 x 256 tiles and of the chunks of K."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def two_norm(a, b):
    return ((a.double() - b).norm() / b.norm()).item()


@pytest.mark.parametrize("M, N, K", [(1, 32, 32), (127, 256, 384), (129, 288, 416), (600, 384, 128), (300, 768, 768), (2000, 768, 3072)])
def test_products(M, N, K):
    import qlka_native
    native = qlka_native.ext()
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x, w, b = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda") / K ** 0.5, torch.randn(N, generator=g, device="cuda")
    lw, lb = torch.rand(K, generator=g, device="cuda") + 0.5, torch.randn(K, generator=g, device="cuda")
    parts = native.split_rows(x, lw, lb, 1e-5)
    h = parts.double().sum(0)
    assert two_norm(h, F.layer_norm(x.double(), (K,), lw.double(), lb.double(), 1e-5)) < 3e-7
    want = h @ w.double().T + b.double()
    torch_err = two_norm(F.linear(h.float(), w, b), want)
    y0 = torch.randn(M, N, generator=g, device="cuda")
    y = y0.clone()
    native.linear_residual(parts, w, b, y)
    assert two_norm(y, want + y0.double()) < max(1.2 * torch_err, 2e-7)
    gelu = native.linear_gelu(parts, w, b).double().sum(0)
    assert two_norm(gelu, F.gelu(want)) < max(1.5 * torch_err, 4e-7)
    assert native.linear_error() == 0


def test_qkv_rotary_layout():
    import qlka_native
    from kernel_attention.encoder import rotary, rotary_angles
    native = qlka_native.ext()
    B, S, H, K = 2, 333, 3, 192
    g = torch.Generator(device="cuda").manual_seed(3)
    x, w, b = torch.randn(B * S, K, generator=g, device="cuda"), torch.randn(3 * H * 64, K, generator=g, device="cuda") / K ** 0.5, torch.randn(3 * H * 64, generator=g, device="cuda")
    parts = native.split_rows(x, torch.ones(K, device="cuda"), torch.zeros(K, device="cuda"), 1e-5)
    table = torch.stack(rotary_angles(S, 32, x.device), dim=-1).contiguous()
    got = native.linear_qkv(parts, w, b, table, B, S, H)
    q, k, v = F.linear(parts.double().sum(0).float(), w, b).view(B, S, 3, H, 64).permute(2, 0, 3, 1, 4)
    for a, want in zip(got, (rotary(q), rotary(k), v)):
        assert two_norm(a, want.double()) < 1e-6


def test_a_kernel_that_gave_up_is_reported():
    """The error word as a kernel would leave it (no kernel is made to give up): the next layer raises, once."""
    import ctypes
    import qlka_native
    from kernel_attention.encoder import Encoder
    word = ctypes.POINTER(ctypes.c_int)()
    assert qlka_native.lib().qlka_linear_error_word(ctypes.byref(word)) == 0
    model = Encoder("add_laplace", layers=1, hidden=128, heads=2, mlp=256, vocab=100).cuda().eval()
    ids = torch.randint(0, 100, (1, 40), device="cuda")
    want = model(ids)
    torch.cuda.synchronize()
    assert word[0] == 0
    word[0] = 1
    with pytest.raises(RuntimeError, match="gave up"):
        model(ids)
    assert word[0] == 0
    word[0] = 1
    assert qlka_native.ext().linear_error() == 1 and qlka_native.ext().linear_error() == 0
    assert torch.equal(model(ids), want)
