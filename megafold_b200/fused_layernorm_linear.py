"""LayerNorm fused into a linear layer, with the module and function interface of the reference.

Mirrors megafold/model/FusedLayernormLinear/fused_layernorm_linear.py: ``LayernormLinear`` (:498-545,
parameters ``WEIGHT[K]``, ``BIAS[K]``, ``linear_weight[K, N]``, ``linear_bias[N]``) and
``LayernormLinearFunction`` (:477-495).  Unlike the reference there is no shape table and no
fallback to torch (:538-541): every shape goes to the CUDA library (``mf_lnl_fwd`` / ``mf_lnl_bwd``).
Row statistics are kept in fp32 (the reference stores them in the input dtype, :361-362).
"""
from __future__ import annotations

import math

import torch
from torch import nn

from . import _lib

__all__ = ["LayernormLinear", "LayernormLinearFunction", "layernorm_linear_forward", "layernorm_linear_backward"]


def layernorm_linear_forward(x, linear_weight, linear_bias, ln_weight, ln_bias, eps: float = 1e-5, flags: int = 0):
    """Returns ``(y [..., N], mean fp32 [M], rstd fp32 [M])``."""
    return _lib.native().lnl_forward(x, linear_weight, linear_bias, ln_weight, ln_bias, eps, flags)


def layernorm_linear_backward(dy, x, linear_weight, ln_weight, ln_bias, mean, rstd, has_linear_bias, flags: int = 0):
    """Returns ``(dx, d_linear_weight, d_linear_bias, d_ln_weight, d_ln_bias)``; parameter gradients fp32."""
    return tuple(_lib.native().lnl_backward(dy, x, linear_weight, ln_weight, ln_bias, mean, rstd, has_linear_bias, flags))


class LayernormLinearFunction(torch.autograd.Function):
    """``apply(X, linear_weight, linear_bias, WEIGHT, BIAS, has_layernorm_bias, has_linear_bias,
    supported_configs)``; the last argument (the reference's Triton tile configs) is ignored.  Under autocast the
    operands are converted to bf16, as the reference's ``custom_fwd(cast_inputs=torch.bfloat16)`` does; the gradients
    come back in the types of the arguments.  The autograd function is native (csrc/torch_ops.cpp); ``forward`` and
    ``backward`` are its two halves, for subclasses."""

    @staticmethod
    @torch.amp.custom_fwd(device_type="cuda", cast_inputs=torch.bfloat16)
    def forward(ctx, X, linear_weight, linear_bias, WEIGHT, BIAS, has_layernorm_bias=True, has_linear_bias=False, supported_configs=None):
        ln_b, lin_b = BIAS if has_layernorm_bias else None, linear_bias if has_linear_bias else None
        y, mean, rstd = layernorm_linear_forward(X, linear_weight, lin_b, WEIGHT, ln_b)
        ctx.save_for_backward(X, linear_weight, lin_b, WEIGHT, ln_b, mean, rstd)
        return y

    @staticmethod
    @torch.amp.custom_bwd(device_type="cuda")
    def backward(ctx, dOUT):
        X, w, b, ln_w, ln_b, mean, rstd = ctx.saved_tensors
        dx, dw, db, d_ln_w, d_ln_b = layernorm_linear_backward(dOUT, X, w, ln_w, ln_b, mean, rstd, b is not None)
        grads = (g if g is None else g.to(t.dtype) for g, t in ((dx, X), (dw, w), (db, b), (d_ln_w, ln_w), (d_ln_b, ln_b)))
        return (*grads, None, None, None)

    @classmethod
    def apply(cls, X, linear_weight, linear_bias, WEIGHT, BIAS, has_layernorm_bias=True, has_linear_bias=False, supported_configs=None):
        if cls is not LayernormLinearFunction:
            return super().apply(X, linear_weight, linear_bias, WEIGHT, BIAS, has_layernorm_bias, has_linear_bias, supported_configs)
        return _lib.native().lnl(X, linear_weight, linear_bias if has_linear_bias else None, WEIGHT, BIAS if has_layernorm_bias else None)


class LayernormLinear(nn.Module):
    """``LayerNorm(K)`` followed by ``Linear(K -> N)`` with the weight stored ``[K, N]``."""

    def __init__(self, K, N, has_layernorm_bias=True, has_linear_bias=True, device=None, dtype=None):
        factory_kwargs = {"device": device, "dtype": dtype}
        super().__init__()
        self.K, self.N = K, N
        self.has_layernorm_bias = has_layernorm_bias
        self.has_linear_bias = has_linear_bias
        self.WEIGHT = nn.Parameter(torch.empty(K, **factory_kwargs))
        self.BIAS = nn.Parameter(torch.empty(K, **factory_kwargs)) if has_layernorm_bias else None
        self.linear_weight = nn.Parameter(torch.empty((K, N), **factory_kwargs))
        self.linear_bias = nn.Parameter(torch.empty((N,), **factory_kwargs)) if has_linear_bias else None
        self.reset_parameters()

    def reset_parameters(self) -> None:
        # same distributions as nn.LayerNorm + nn.Linear (Kaiming-uniform on the [N, K] view)
        nn.init.ones_(self.WEIGHT)
        if self.BIAS is not None:
            nn.init.zeros_(self.BIAS)
        with torch.no_grad():
            as_linear = torch.empty((self.N, self.K), device=self.linear_weight.device, dtype=self.linear_weight.dtype)
            nn.init.kaiming_uniform_(as_linear, a=math.sqrt(5))
            self.linear_weight.copy_(as_linear.T)
        if self.linear_bias is not None:
            bound = 1 / math.sqrt(self.K) if self.K > 0 else 0
            nn.init.uniform_(self.linear_bias, -bound, bound)

    def forward(self, X):
        return LayernormLinearFunction.apply(X, self.linear_weight, self.linear_bias, self.WEIGHT, self.BIAS,
                                             self.has_layernorm_bias, self.has_linear_bias, None)

    def extra_repr(self):
        return f"K={self.K}, N={self.N}, has_linear_bias={self.has_linear_bias}"
