"""Performance cases of the library: what a program built on it has it do, through its public entry points.

A case is a dict of plain values; `call` names the entry point:

  attention        kernel_attention.attention(q, k, v, kernel, tau, keep)   inference
  attention_train  the same under autograd, with the gradients of q, k and v
  laplace          weighted_laplace_sum                                     forward
  abs              weighted_abs_sum_full                                    forward
  abs_train        weighted_abs_sum_full, forward and backward
  sgn              weighted_sgn_sum
  encoder          the 12-layer pre-LN encoder on token ids

Sizes: B batch, H heads, N keys, M queries (attention: M = N), D features, C value channels. The ranges are those of the
benchmark configurations (256 to 262144 keys, 1 to 256 heads), of the speed-and-memory sweep (2^7 to 2^17 keys at 4 x 12 heads)
and of the tests (lengths and channel counts that are no multiple of anything).
"""

import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "quasi-linear-kernel-attention_b200"))

from kernel_attention.attention import attention  # noqa: E402
from kernel_attention.encoder import Encoder  # noqa: E402
from weighted_abs_sum import weighted_abs_sum_full, weighted_sgn_sum  # noqa: E402
from weighted_laplace_sum import weighted_laplace_sum  # noqa: E402

HIDDEN, HEADS, MLP, VOCAB, LAYERS = 768, 12, 3072, 30528, 12      # the encoder of the benchmark configuration


def _attn(call, kernel, B, H, N, D, C, tau, masked=False, scale=1.0, uniform=False):
    return {"call": call, "kernel": kernel, "B": B, "H": H, "N": N, "M": N, "D": D, "C": C, "tau": tau, "masked": masked,
            "scale": scale, "uniform": uniform}


def _op(call, B, H, N, M, D, C, scale=1.0):
    return {"call": call, "B": B, "H": H, "N": N, "M": M, "D": D, "C": C, "scale": scale, "uniform": False}


def listed():
    cases = [
        # the shortest sequence of the sweep: a call that is all latency
        ("short_riesz", _attn("attention", "add_riesz", 4, 12, 128, 64, 64, 1.0)),
        # one small head group at a moderate length, as in a first experiment or a single request
        ("small_laplace", _attn("attention", "add_laplace", 1, 4, 1024, 32, 32, 1.0)),
        # many short sequences with one head, values spread over several bump widths
        ("batch_bump", _attn("attention", "add_bump", 256, 1, 600, 64, 64, 1.0, scale=3.0, uniform=True)),
        # a padded batch of ragged texts: odd length, key-keep mask
        ("padded_laplace", _attn("attention", "add_laplace", 8, 12, 777, 64, 64, 0.5, masked=True)),
        # a training step of a small model
        ("train_laplace", _attn("attention_train", "add_laplace", 4, 12, 1024, 64, 64, 0.5)),
        # the abs-sum training step of the benchmark
        ("train_abs", _op("abs_train", 8, 12, 4096, 4096, 64, 64, scale=0.5)),
        # the signed sum on sizes that are no multiple of anything, more keys than queries
        ("ragged_sgn", _op("sgn", 2, 12, 3001, 1777, 48, 40)),
        # few queries against many keys with wide values (pooling, cross-attention)
        ("cross_laplace", _op("laplace", 1, 16, 8191, 1030, 64, 128)),
        # the headline workload
        ("laplace_16384", _op("laplace", 4, 12, 16384, 16384, 64, 64, scale=2.0)),
        # long context
        ("laplace_65536", _op("laplace", 1, 16, 65536, 65536, 64, 64)),
        ("abs_262144", _op("abs", 1, 16, 262144, 262144, 64, 64)),
        # the end-to-end encoder of the benchmark configuration
        ("encoder", {"call": "encoder", "kernel": "add_laplace", "B": 2, "N": 8192}),
    ]
    return [dict(c, name=name) for name, c in cases]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: lengths over their logarithm, heads so that the whole stays under the largest listed case."""
    call = rng.choices(["attention", "attention_train", "laplace", "abs", "abs_train", "sgn", "encoder"], [8, 4, 3, 2, 2, 1, 1])[0]
    if call == "encoder":
        n = _log(rng, 128, 8192)
        return {"call": call, "kernel": "add_laplace", "B": rng.randint(1, max(1, min(16, 16384 // n))), "N": n}
    D = rng.choice([16, 32, 48, 64, 64, 64, 96])
    C = rng.choice([16, 32, 33, 40, 64, 64, 64, 96, 128])
    train = call in ("attention_train", "abs_train")
    N = _log(rng, 64, 16384 if train or call == "sgn" else 65536)
    most = max(1, min(256, 2 ** (25 if train else 26) // (N * max(D, C))))
    heads = _log(rng, 1, most)
    H = rng.choice([h for h in (1, 2, 3, 4, 8, 12, 16) if h <= heads])
    B = heads // H
    if call.startswith("attention"):
        kernel = rng.choice(["add_laplace", "add_laplace", "add_riesz", "add_bump"])
        tau = {"add_laplace": 0.5, "add_riesz": 1.0, "add_bump": 1.5}[kernel]
        return _attn(call, kernel, B, H, N, D, C, tau, masked=rng.random() < 0.4, scale=rng.choice([0.5, 1.0, 2.0]), uniform=rng.random() < 0.2)
    M = N if rng.random() < 0.6 else max(1, min(N, _log(rng, 64, 65536)))
    return _op(call, B, H, N, M, D, C, scale=rng.choice([0.5, 1.0, 2.0]))


def _points(case, shape, gen):
    if case["uniform"]:
        return (torch.rand(*shape, generator=gen, device="cuda") * 2.0 - 1.0) * case["scale"]
    return torch.randn(*shape, generator=gen, device="cuda") * case["scale"]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = {"case": case}
    if case["call"] == "encoder":
        torch.manual_seed(seed)
        with torch.device("cuda"):
            state["model"] = Encoder(case["kernel"], layers=LAYERS, hidden=HIDDEN, heads=HEADS, mlp=MLP, vocab=VOCAB).eval()
        state["ids"] = torch.randint(0, VOCAB, (case["B"], case["N"]), generator=gen, device="cuda")
        return state
    B, H, N, M, D, C = (case[x] for x in "BHNMDC")
    if case["call"].startswith("attention"):
        state["q"], state["k"] = _points(case, (B, H, N, D), gen), _points(case, (B, H, N, D), gen)
        state["v"] = torch.randn(B, H, N, C, generator=gen, device="cuda")
        state["keep"] = None
        if case["masked"]:      # texts of different lengths, padded at the end
            length = torch.randint(max(1, N // 2), N + 1, (B, 1), generator=gen, device="cuda")
            state["keep"] = torch.arange(N, device="cuda")[None, :] < length
        if case["call"] == "attention_train":
            state["g"] = torch.randn(B, H, N, C, generator=gen, device="cuda")
    else:
        P = B * H
        state["q"], state["k"] = _points(case, (P, D, M), gen), _points(case, (P, D, N), gen)
        state["v"] = torch.randn(P, N, C, generator=gen, device="cuda")
        if case["call"] in ("abs_train", "sgn"):
            state["g"] = torch.randn(P, M, C, generator=gen, device="cuda")
        if case["call"] == "abs_train":
            state["g_u"] = torch.randn(P, M, generator=gen, device="cuda")
    if case["call"] in ("attention_train", "abs_train"):
        for x in "qkv":
            state[x].requires_grad_(True)
    return state


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "encoder":
        return state["model"](state["ids"])
    q, k, v = state["q"], state["k"], state["v"]
    if call == "attention":
        return attention(q, k, v, case["kernel"], case["tau"], state["keep"])
    if call == "attention_train":
        out = attention(q, k, v, case["kernel"], case["tau"], state["keep"])
        return out, torch.autograd.grad(out, (q, k, v), state["g"])
    if call == "laplace":
        return weighted_laplace_sum(q, k, v)
    if call == "abs":
        return weighted_abs_sum_full(q, k, v)
    if call == "abs_train":
        out = weighted_abs_sum_full(q, k, v)
        return out, torch.autograd.grad(out, (q, k, v), (state["g"], state["g_u"]))
    return weighted_sgn_sum(q, k, v, state["g"])


def _sums(P, N, M, D, C, kernel_sums):
    """Operations of the sorted evaluation: per feature, key and channel the running sums, per feature, query and channel their use."""
    return P * D * C * (4 * N + 4 * M * kernel_sums)


def work(case):
    if case["call"] == "encoder":
        B, N = case["B"], case["N"]
        weights = LAYERS * (4 * HIDDEN * HIDDEN + 2 * HIDDEN * MLP + 9 * HIDDEN + MLP) + B * N * HIDDEN + 2 * HIDDEN
        gemm = 2 * B * N * LAYERS * (4 * HIDDEN * HIDDEN + 2 * HIDDEN * MLP)
        d = HIDDEN // HEADS
        return {"bytes": 4 * (weights + B * N * HIDDEN) + 8 * B * N, "flops": gemm + LAYERS * _sums(B * HEADS, N, N, d, d, 1)}
    P, N, M, D, C = case["B"] * case["H"], case["N"], case["M"], case["D"], case["C"]
    q, k, v, out = P * M * D, P * N * D, P * N * C, P * M * C
    sums = 3 if case.get("kernel") == "add_bump" else 1
    call = case["call"]
    if call == "attention":
        return {"bytes": 4 * (q + k + v + out) + (case["B"] * N if case["masked"] else 0), "flops": _sums(P, N, M, D, C, sums)}
    if call == "attention_train":
        return {"bytes": 4 * (2 * (q + k + v) + 2 * out) + (case["B"] * N if case["masked"] else 0), "flops": 4 * _sums(P, N, M, D, C, sums)}
    if call in ("laplace", "abs"):
        return {"bytes": 4 * (q + k + v + out + P * M), "flops": _sums(P, N, M, D, C, 1)}
    if call == "abs_train":
        return {"bytes": 4 * (2 * (q + k + v) + 2 * out + 2 * P * M), "flops": 4 * _sums(P, N, M, D, C, 1)}
    return {"bytes": 4 * (q + k + v + out + q), "flops": _sums(P, N, M, D, C, 1)}


def tolerance(case):
    """fp32 sums in any order. The Laplace recurrence multiplies as many step decays as there are keys, each rounded once, so its
    error grows with the length. The attention kernels around the abs sum subtract sums that are larger than their result, the
    more so the longer the sequence."""
    n = case["N"]
    if case["call"] == "encoder":
        return {"rel": 5e-5}
    if case.get("kernel", "add_laplace") != "add_laplace":
        return {"rel": 2e-5 if n <= 16384 else 1e-4}
    if case["call"].startswith(("laplace", "attention")):
        return {"rel": max(1e-5, 1e-9 * n)}
    return {"rel": 1e-5}
