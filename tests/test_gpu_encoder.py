"""The end-to-end encoder harness (the 12-layer pre-LN encoder, shrunk): the add_laplace encoder output equals
the same network with its attention evaluated by the float64 O(N^2) oracle, and the native blocks compute what calling the
torch modules one by one does, hooks, replacements and casts included."""

import pytest
import torch
import torch.nn as nn

from oracle import direct

pytestmark = pytest.mark.gpu


def test_encoder_matches_checker_attention():
    import importlib
    am = importlib.import_module("kernel_attention.attention")      # the module (the package also exports the function)
    from kernel_attention.encoder import Encoder
    torch.manual_seed(0)
    model = Encoder("add_laplace", layers=2, hidden=128, heads=2, mlp=256, vocab=1000).cuda().eval()
    ids = torch.randint(0, 1000, (2, 300), device="cuda")
    got = model(ids)
    real = am.attention
    try:
        am.attention = lambda q, k, v, kernel, tau, keep=None: direct.attention(q.cpu(), k.cpu(), v.cpu(), kernel, tau, keep).float().cuda()
        want = model(ids)
    finally:
        am.attention = real
    assert got.shape == (2, 300, 128)
    assert (got - want).abs().max().item() < 1e-3 * want.abs().max().item()


def test_measure_runs_small():
    from kernel_attention.encoder import measure
    ms, mib = measure("add_laplace", batch=1, seq=512, layers=2, reps=1)
    assert ms > 0 and mib > 0


def small(kernel="add_laplace"):
    from kernel_attention.encoder import Encoder
    torch.manual_seed(0)
    return Encoder(kernel, layers=2, hidden=128, heads=2, mlp=256, vocab=100).cuda().eval(), torch.randint(0, 100, (2, 65), device="cuda")


def module_by_module(model, ids, keep=None):
    with torch.no_grad():
        x = model.embed(ids)
        for block in model.blocks:
            x = block(x, keep)
        return model.ln(x)


class Doubled(nn.Linear):
    def forward(self, x):
        return 2 * super().forward(x)


CHANGES = {
    "none": lambda b: None,
    "forward hook": lambda b: b.qkv.register_forward_hook(lambda m, i, o: 2 * o),
    "forward pre-hook": lambda b: b.fc2.register_forward_pre_hook(lambda m, i: (2 * i[0],)),
    "hook on the block": lambda b: b.register_forward_hook(lambda m, i, o: 2 * o),
    "another linear class": lambda b: setattr(b, "proj", Doubled(128, 128).cuda()),
    "no bias": lambda b: setattr(b, "fc1", nn.Linear(128, 256, bias=False).cuda()),
    "no layer norm weight": lambda b: setattr(b, "ln2", nn.LayerNorm(128, elementwise_affine=False)),
    "forward of the instance": lambda b: setattr(b.fc1, "forward", lambda x: 3 * nn.functional.linear(x, b.fc1.weight, b.fc1.bias)),
}


@pytest.mark.parametrize("change", CHANGES)
def test_native_blocks_equal_the_modules(change):
    model, ids = small()
    CHANGES[change](model.blocks[0])
    x = model.embed(ids)
    assert [block.fits_native(x) for block in model.blocks] == [change == "none", True]
    keep = torch.ones(2, 65, dtype=torch.bool, device="cuda")
    keep[1, 40:] = False
    for mask in (None, keep):
        got, want = model(ids, mask), module_by_module(model, ids, mask)
        # (two layers of fp32 products and sums in other orders, about 1e-6; any of the changes moves the output by more than 1e-2)
        assert ((got - want).norm() / want.norm()).item() < 1e-5


def test_casts_modes_and_precision_settings_reach_the_modules():
    model, ids = small("softmax")
    with torch.autocast("cuda", torch.bfloat16):
        assert torch.equal(model(ids), module_by_module(model, ids))
    from torch.utils.flop_counter import FlopCounterMode
    with FlopCounterMode(display=False) as count:
        model(ids)
    assert count.get_total_flops() >= 2 * 2 * 130 * (4 * 128 * 128 + 2 * 128 * 256)
    try:
        torch.backends.cuda.matmul.fp32_precision = "tf32"
        assert torch.equal(model(ids), module_by_module(model, ids))
    finally:
        torch.backends.cuda.matmul.fp32_precision = "none"


def test_tensors_seen_by_hooks_stay_as_they_were():
    """The native block works in place: on a copy where a hook can have kept its input."""
    for where in ("embed", "block"):
        model, ids = small()
        kept = []
        (model.embed if where == "embed" else model.blocks[0]).register_forward_hook(lambda m, i, o: kept.append((o, o.clone())))
        model(ids)
        assert torch.equal(*kept[0])


@pytest.mark.filterwarnings("ignore")
def test_traced_and_compiled_models_hold_the_whole_computation():
    from torch.fx.experimental.proxy_tensor import make_fx
    model, ids = small("softmax")
    other = ids.flip(0).flip(1).contiguous()
    want = module_by_module(model, other)
    for made in (torch.jit.trace(model, (ids,), check_trace=False), torch.compile(model, backend="eager", fullgraph=True), make_fx(model)(ids)):
        assert ((made(other) - want).norm() / want.norm()).item() < 1e-5
    assert ((torch.func.vmap(model)(other[:, None])[:, 0] - want).norm() / want.norm()).item() < 1e-5
