"""SwiGLU and the fused Transition block with the module interface of the reference.

Mirrors megafold/model/FusedTransition/fused_transition.py: ``FusedSwiGLUFunction`` / ``FusedSwiGLU``
(:96-116) and ``FusedTransition`` (:118-151).  ``FusedTransition`` keeps the reference's ``ff``
``nn.Sequential`` so that ``state_dict`` keys are unchanged (``ff.0.WEIGHT``, ``ff.0.BIAS``,
``ff.0.linear_weight``, ``ff.2.weight``), but its forward runs LN -> Linear -> SwiGLU -> Linear as one
operator (``mf_transition_fwd`` / ``mf_transition_bwd``) that does not keep the hidden activations:
backward recomputes them from ``x``.  SwiGLU backward writes to a new buffer (the reference
overwrites its saved input, :49-52).
"""
from __future__ import annotations

import torch
from torch import nn

from . import _lib
from .fused_layernorm_linear import LayernormLinear

__all__ = ["FusedSwiGLUFunction", "FusedSwiGLU", "FusedTransition", "TransitionFunction",
           "transition_forward", "transition_backward"]


class FusedSwiGLUFunction(torch.autograd.Function):
    """``apply(x [..., 2 * inner])``; the autograd function is native (csrc/torch_ops.cpp).  ``forward`` and ``backward``
    are its two halves, for subclasses."""

    @staticmethod
    @torch.amp.custom_fwd(device_type="cuda", cast_inputs=torch.bfloat16)
    def forward(ctx, input):
        ctx.save_for_backward(input)
        return _lib.native().swiglu(input)

    @staticmethod
    @torch.amp.custom_bwd(device_type="cuda")
    def backward(ctx, grad_output):
        x = ctx.saved_tensors[0].detach().requires_grad_(True)
        with torch.enable_grad():
            y = _lib.native().swiglu(x)
        return torch.autograd.grad(y, x, grad_output.to(y.dtype))[0]

    @classmethod
    def apply(cls, input):
        return _lib.native().swiglu(input) if cls is FusedSwiGLUFunction else super().apply(input)


class FusedSwiGLU(nn.Module):
    def forward(self, x):
        return FusedSwiGLUFunction.apply(x)


def transition_forward(x, ln_weight, ln_bias, w1, w2, eps: float = 1e-5, flags: int = 0):
    """``w1`` [dim, 2*inner], ``w2`` [dim, inner].  Returns ``(y, mean, rstd)``."""
    return _lib.native().transition_forward(x, ln_weight, ln_bias, w1, w2, eps, flags)


def transition_backward(dy, x, ln_weight, ln_bias, w1, w2, mean, rstd, flags: int = 0):
    """Returns ``(dx, d_ln_weight, d_ln_bias, dw1, dw2)``; parameter gradients fp32."""
    return tuple(_lib.native().transition_backward(dy, x, ln_weight, ln_bias, w1, w2, mean, rstd, flags))


class TransitionFunction(torch.autograd.Function):
    """``apply(x, ln_weight | None, ln_bias | None, w1 [dim, 2*inner], w2 [dim, inner])``; the autograd function is native
    (csrc/torch_ops.cpp).  ``forward`` and ``backward`` are its two halves, for subclasses."""

    @staticmethod
    @torch.amp.custom_fwd(device_type="cuda", cast_inputs=torch.bfloat16)
    def forward(ctx, x, ln_weight, ln_bias, w1, w2):
        y, mean, rstd = transition_forward(x, ln_weight, ln_bias, w1, w2)
        ctx.save_for_backward(x, ln_weight, ln_bias, w1, w2, mean, rstd)
        return y

    @staticmethod
    @torch.amp.custom_bwd(device_type="cuda")
    def backward(ctx, dy):
        x, ln_weight, ln_bias, w1, w2, mean, rstd = ctx.saved_tensors
        grads = transition_backward(dy, x, ln_weight, ln_bias, w1, w2, mean, rstd)
        return tuple(g if g is None else g.to(t.dtype) for g, t in zip(grads, (x, ln_weight, ln_bias, w1, w2)))

    @classmethod
    def apply(cls, x, ln_weight, ln_bias, w1, w2):
        if cls is not TransitionFunction:
            return super().apply(x, ln_weight, ln_bias, w1, w2)
        return _lib.native().transition(x, ln_weight, ln_bias, w1, w2)


class FusedTransition(nn.Module):
    def __init__(self, dim, expansion_factor=4, include_ln=True, use_layernormlinear=True, device=None, dtype=None):
        factory_kwargs = {"device": device, "dtype": dtype}
        super().__init__()
        self.dim = dim
        dim_inner = int(dim * expansion_factor)
        self.dim_inner = dim_inner
        self.include_ln = include_ln
        self.use_layernormlinear = use_layernormlinear
        if include_ln:
            if use_layernormlinear:
                self.ff = nn.Sequential(
                    LayernormLinear(dim, dim_inner * 2, has_linear_bias=False, **factory_kwargs),
                    FusedSwiGLU(),
                    nn.Linear(dim_inner, dim, bias=False, **factory_kwargs),
                )
            else:
                self.ff = nn.Sequential(
                    nn.LayerNorm(dim, **factory_kwargs),
                    nn.Linear(dim, dim_inner * 2, bias=False, **factory_kwargs),
                    FusedSwiGLU(),
                    nn.Linear(dim_inner, dim, bias=False, **factory_kwargs),
                )
        else:
            self.ff = nn.Sequential(
                nn.Linear(dim, dim_inner * 2, bias=False, **factory_kwargs),
                FusedSwiGLU(),
                nn.Linear(dim_inner, dim, bias=False, **factory_kwargs),
            )

    def forward(self, input):
        if self.include_ln and self.use_layernormlinear:
            lnl = self.ff[0]
            return TransitionFunction.apply(input, lnl.WEIGHT, lnl.BIAS, lnl.linear_weight, self.ff[2].weight)
        if self.include_ln:
            ln, lin = self.ff[0], self.ff[1]
            return TransitionFunction.apply(input, ln.weight, ln.bias, lin.weight.t(), self.ff[3].weight)
        return TransitionFunction.apply(input, None, None, self.ff[0].weight.t(), self.ff[2].weight)

    def extra_repr(self):
        return f"dim={self.dim}, dim_inner={self.dim_inner}"
