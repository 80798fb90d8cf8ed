"""Normalised additive-kernel attention on (B, H, S, D) fp32 CUDA tensors for the three kernels whose
efficient evaluation goes through the sorted-walk operators: add_laplace, add_riesz, add_bump.

`attention(q, k, v, kernel, tau, keep=None)` answers the same call as the reference's
`attention(..., impl="efficient")` (Experiments/kernel_attention/attention.py:95-126) for those kernels;
the reference's own file also runs unchanged on top of the two operator packages of this library.

Two routes:
* one native call forward and, where gradients are wanted, one backward (`qlka_native.attention`): layout change, tau,
  masking, the sums and the normalisation all happen inside the library;
* the cases without such a call (gradients of add_riesz and add_bump at long lengths, add_bump beyond 5461 keys, training with a
  temperature that is a tensor to broadcast or to train, or that is not above 0, or with a mask that wants a gradient; calls that
  torch.jit.trace records) - the sums are assembled here from the differentiable operators. Every kernel is described
  by two small functions: `sums` returns the unnormalised numerator sum_j A_ij v_j and row sum sum_j A_ij over
  ALL S keys, and `at_origin` returns A(q_i, 0), the weight a key placed at the origin has. Masked keys are moved
  to the origin with a zero value row, so they add nothing to the numerator and exactly `at_origin` each to the
  row sum, which is subtracted again. Where a query coordinate lies on a kink there, `at_origin` has the operators' derivative
  (of |q - k| with respect to q: -1 at 0), not torch's, so that the gradients cancel too.
"""

import torch

import qlka_native as _native
from weighted_abs_sum import weighted_abs_sum_full
from weighted_laplace_sum import weighted_laplace_sum

EPS = 1e-3        # offset of the Riesz kernel (Experiments/kernel_attention/kernels.py:9)
CLAMP = 1e-6      # floor of the row sum (Experiments/kernel_attention/attention.py:21)
TAU = {"add_laplace": 0.5, "add_riesz": 1.0, "add_bump": 1.5}   # default temperatures, kernels.py:13-25


# ---- add_laplace: A_ij = sum_d exp(-|q_id - k_jd|)
def _laplace_sums(q, k, v):
    return weighted_laplace_sum(q, k, v)


def _laplace_at_origin(q):
    return torch.exp(torch.where(q > 0, -q, q)).sum(dim=1)


# ---- add_riesz: A_ij = |q_i|_1 + |k_j|_1 - |q_i - k_j|_1 + EPS; the two norms are rank-1 terms around the abs sum
def _riesz_sums(q, k, v):
    dist_v, dist_1 = weighted_abs_sum_full(q, k, v)
    q_norm = q.abs().sum(dim=1) + EPS                     # (P, S)   the offset rides with the query norm
    k_norm = k.abs().sum(dim=1)                           # (P, S)
    v_total = v.sum(dim=1)                                # (P, C)
    kv_total = torch.einsum("ps,psc->pc", k_norm, v)      # (P, C)
    num = q_norm.unsqueeze(2) * v_total.unsqueeze(1) + kv_total.unsqueeze(1) - dist_v
    row = q_norm * k.shape[2] + k_norm.sum(dim=1, keepdim=True) - dist_1
    return num, row


class _RieszAtOrigin(torch.autograd.Function):
    """The norm of q cancels against |q - 0|_1, the derivatives (0 and -1 where q is 0) do not. (As a node of its own it costs a masked
    training step of 4 heads x 5000 2 %, composed of torch's operations 6 %.)"""

    @staticmethod
    def forward(ctx, q):
        ctx.save_for_backward(q)
        return torch.full_like(q[:, 0, :], EPS)

    @staticmethod
    def backward(ctx, g):
        return torch.where(ctx.saved_tensors[0] == 0, g.unsqueeze(1), 0.0)


# ---- add_bump: A_ij = sum_d max(0, 1 - |x|), x = q_id - k_jd, and max(0, 1 - |x|) = (|x + 1| + |x - 1|) / 2 - |x|
_BUMP_TERMS = ((0.0, -1.0), (1.0, 0.5), (-1.0, 0.5))      # (query shift, weight) of the three abs sums


def _bump_sums(q, k, v):
    num = row = None
    for shift, weight in _BUMP_TERMS:
        dist_v, dist_1 = weighted_abs_sum_full(q + shift if shift else q, k, v)
        num = weight * dist_v if num is None else num + weight * dist_v
        row = weight * dist_1 if row is None else row + weight * dist_1
    return num, row


class _BumpAtOrigin(torch.autograd.Function):
    """sum_d max(0, 1 - |q_d|) with the derivative of the three terms: 1 for q in (-1, 0], -1 in (0, 1], else 0."""

    @staticmethod
    def forward(ctx, q):
        ctx.save_for_backward(q)
        return (1.0 - q.abs()).clamp_min(0.0).sum(dim=1)

    @staticmethod
    def backward(ctx, g):
        step, g = ctx.saved_tensors[0].ceil(), g.unsqueeze(1)
        return torch.where(step == 0, g, torch.where(step == 1, -g, 0.0))


_ROUTES = {"add_laplace": (_laplace_sums, _laplace_at_origin),
           "add_riesz": (_riesz_sums, _RieszAtOrigin.apply),
           "add_bump": (_bump_sums, _BumpAtOrigin.apply)}


def _needs_operators(q, k, v, tau, keep):
    """Whether a call asks for gradients that the native backward pass does not give, for a temperature it does not take, or for a record."""
    if torch.jit.is_tracing():
        return True
    by_tensor = isinstance(tau, torch.Tensor)
    trained = (by_tensor and tau.requires_grad) or (keep is not None and keep.requires_grad)
    if not (trained or q.requires_grad or k.requires_grad or v.requires_grad) or not torch.is_grad_enabled():
        return False
    return trained or (by_tensor and tau.numel() != 1) or not tau > 0


def attention(q, k, v, kernel, tau, keep=None):
    """q, k (B, H, S, D), v (B, H, S, Dv) fp32 CUDA; keep (B, S) bool/float key-keep mask or None -> (B, H, S, Dv)."""
    assert q.dtype == k.dtype == v.dtype == torch.float32, "kernel attention runs in fp32 only"
    if kernel not in _ROUTES:
        raise ValueError(f"kernel must be one of {tuple(_ROUTES)}, got {kernel!r}")
    B, H, S, D = q.shape
    if (kernel != "add_bump" or 3 * S <= 16384) and not _needs_operators(q, k, v, tau, keep):      # the fused add_bump shares one shared-memory sort between its three shifts
        out = _native.attention(kernel, q, k, v, tau, keep)
        if out is not None:
            return out

    sums, at_origin = _ROUTES[kernel]
    heads = B * H
    qs = (q / tau).permute(0, 1, 3, 2).reshape(heads, D, S).contiguous()          # (P, D, S): one sorted axis per feature
    ks = (k / tau).permute(0, 1, 3, 2).reshape(heads, D, S)
    vs = v.reshape(heads, S, v.shape[3])
    if keep is not None:
        kept = keep.to(q.dtype).repeat_interleave(H, dim=0)                       # (P, S)
        if keep.dtype != torch.bool:
            ks, vs = ks * kept.unsqueeze(1), vs * kept.unsqueeze(2)
        on = kept != 0                                                            # (whatever stands elsewhere: 0 times NaN would be NaN)
        ks, vs = torch.where(on.unsqueeze(1), ks, 0.0), torch.where(on.unsqueeze(2), vs, 0.0)
    num, row = sums(qs, ks.contiguous(), vs.contiguous())
    if keep is not None:
        row = row - (S - kept.sum(dim=1, keepdim=True)) * at_origin(qs)
    return (num / row.clamp_min(CLAMP).unsqueeze(2)).view(B, H, S, -1)
