"""Pair-biased, key-masked attention with the call signature of the reference's ``TritonEvoformer``.

Mirrors ``EvoformerAttention`` / ``TritonEvoformer`` of
megafold/model/FusedEvoAttention/evoattention.py:688-905: five positional tensors
``(Q, K, V, res_mask, pair_bias)``, output ``[B, N, L, H, D]``, gradients
``(dQ, dK, dV, None, d_pair_bias)``.  The work is done by the CUDA library behind the C ABI
(``mf_evo_fwd`` / ``mf_evo_bwd``); tensors on any other device are rejected.

Differences from the reference, all on purpose:
  * no transposed copies: the kernels read and write the ``[B, N, L, H, D]`` layout directly and
    accept strided q/k/v;
  * a boolean (or uint8) ``res_mask`` is a keep-mask with the semantics of the reference's PyTorch
    attention (``masked_fill(~mask, -finfo.max)``, megafold/model/attention.py:522-524); a floating
    ``res_mask`` is added to the logits, which is what the reference kernel does (evoattention.py:66);
  * ``d_pair_bias`` is accumulated in fp32 in a fixed order on every kernel path (bit-reproducible; the
    reference adds rows with atomics, evoattention.py:465) and returned in ``pair_bias.dtype``; the reference
    rounds it to ``dO.dtype`` first (evoattention.py:903).  ``dQ`` is bit-reproducible too unless the
    tensor-core path has to sum partial rows with fp32 atomics (very few rows, or L > 768).
"""
from __future__ import annotations

import torch

from . import _lib

__all__ = ["EvoformerAttention", "TritonEvoformer", "evo_attention_forward", "evo_attention_backward"]


def _check_shapes(q, k, v, res_mask, pair_bias):
    """Returns ``(B, N, L, H, D)``; raises ValueError / TypeError when the five tensors do not fit together."""
    return _lib.native().check_shapes(q, k, v, res_mask, pair_bias)


def _fill_common(a, q, k, v, res_mask, pair_bias, flags):
    """Fills the ctypes structure of an entry point that has no torch function (``mf_evo_bwd_noalloc``)."""
    B, N, L, H, D = q.shape
    a.B, a.N, a.L, a.H, a.D = B, N, L, H, D
    a.dtype = _lib.dtype_code(q.dtype)
    a.bias_dtype = _lib.dtype_code(pair_bias.dtype)
    a.mask_dtype = _lib.dtype_code(res_mask.dtype)
    a.flags = flags
    a.q, a.k, a.v = q.data_ptr(), k.data_ptr(), v.data_ptr()
    a.q_strides[:] = q.stride()
    a.k_strides[:] = k.stride()
    a.v_strides[:] = v.stride()
    m = res_mask.expand(B, N, 1, 1, L)
    a.mask = m.data_ptr()
    a.mask_strides[:] = (m.stride(0), m.stride(1), m.stride(4))
    pb = pair_bias.expand(B, 1, H, L, L)
    a.bias = pb.data_ptr()
    a.bias_strides[:] = (pb.stride(0), pb.stride(2), pb.stride(3), pb.stride(4))


def evo_attention_forward(q, k, v, res_mask, pair_bias, flags: int = 0):
    """Returns ``(O [B,N,L,H,D], LSE fp32 [B,N,H,L])``; ``mf_evo_fwd`` of the C ABI."""
    return _lib.native().evo_forward(q, k, v, res_mask, pair_bias, flags)


def evo_attention_backward(d_o, q, k, v, res_mask, pair_bias, o, lse, flags: int = 0, dbias_ready=None):
    """Returns ``(dQ, dK, dV, dBias)``; dBias has ``pair_bias``'s shape and dtype. ``mf_evo_bwd``.

    ``dbias_ready``: an optional ``torch.cuda.Event`` that the library records on the current stream as soon as dBias is
    final (before dQ / dK / dV on the tensor-core path), for callers that reduce dBias over row shards on another stream."""
    event = 0
    if dbias_ready is not None:
        with torch.cuda.device(q.device):
            dbias_ready.record()                     # creates the underlying cudaEvent_t; the library records it again
        event = dbias_ready.cuda_event
    return _lib.native().evo_backward(d_o, q, k, v, res_mask, pair_bias, o, lse, flags, event)


def TritonEvoformer(Q, K, V, res_mask, pair_bias):
    """Q, K, V: [Batch, N_seq, N_res, Head, Dim]; res_mask: [Batch, N_seq, 1, 1, N_res];
    pair_bias: [Batch, 1, Head, N_res, N_res] (shared by the N_seq rows)."""
    return _lib.native().evo_attention(Q, K, V, res_mask, pair_bias)


class EvoformerAttention(torch.autograd.Function):
    """The operator under the reference's class name: ``EvoformerAttention.apply`` is ``TritonEvoformer``, whose autograd
    function is native (csrc/torch_ops.cpp).  ``forward`` and ``backward`` are its two halves, for subclasses."""

    @staticmethod
    def forward(ctx, Q, K, V, res_mask, pair_bias):
        o, lse = evo_attention_forward(Q, K, V, res_mask, pair_bias)
        ctx.save_for_backward(Q, K, V, res_mask, pair_bias, o, lse)
        return o

    @staticmethod
    def backward(ctx, dO):
        Q, K, V, res_mask, pair_bias, o, lse = ctx.saved_tensors
        dq, dk, dv, d_bias = evo_attention_backward(dO, Q, K, V, res_mask, pair_bias, o, lse)
        return dq, dk, dv, None, d_bias

    @classmethod
    def apply(cls, *args):
        return TritonEvoformer(*args) if cls is EvoformerAttention else super().apply(*args)
