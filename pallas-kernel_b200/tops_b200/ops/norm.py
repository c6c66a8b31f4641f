"""Row normalisations next to the attention kernels:

* `l2norm(x, eps=1e-6)`: `x / sqrt(sum(x^2) + eps)` over the last dimension, the q/k normalisation of
  KDA (`tops/cpu/ops/kda/fused_recurrent.py:14-18`);
* `FusedRMSNormGated`: `RMSNorm(x) * weight * silu(g)` (`tops/modules/fused_norm_gate.py:6-37`), the norm
  the reference applies to the attention output.

Both are differentiable; each direction is one kernel (plus a small fixed-order sum for the weight
gradient).  The last dimension must be a multiple of 4 and at most 1024.
"""
from __future__ import annotations

import torch

from .._lib import ops_ext as X
from ._recorded import call


def _check(x):
    D = x.shape[-1]
    assert D % 4 == 0 and 0 < D <= 1024, f"last dimension must be a multiple of 4 and <= 1024, got {D}"


def l2norm(x, eps=1e-6):
    """x / sqrt(sum(x^2, -1) + eps), in x's dtype (fp32 arithmetic)."""
    _check(x)
    return call(X.l2norm, x, float(eps))


def rmsnorm_gated(x, g, weight=None, eps=1e-5):
    """x * rsqrt(mean(x^2, -1) + eps) * weight * silu(g) in x's dtype (fp32 arithmetic)."""
    _check(x)
    assert g.shape == x.shape, f"g shape {tuple(g.shape)} != x shape {tuple(x.shape)}"
    assert weight is None or weight.numel() == x.shape[-1], f"weight shape {tuple(weight.shape)} != ({x.shape[-1]},)"
    return call(X.rmsnorm_gated, x, g, weight, float(eps))


class FusedRMSNormGated(torch.nn.Module):
    """RMSNorm + SiLU gate (`tops/modules/fused_norm_gate.py:6-37`): `output = RMSNorm(x) * silu(g)`."""

    def __init__(self, hidden_size: int, elementwise_affine: bool = True, eps: float = 1e-5, device=None):
        super().__init__()
        self.hidden_size, self.eps = hidden_size, eps
        self.weight = torch.nn.Parameter(torch.ones(hidden_size, device=device)) if elementwise_affine else None

    def forward(self, x, g):
        return rmsnorm_gated(x, g, self.weight, self.eps)
