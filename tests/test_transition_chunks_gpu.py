"""Fused Transition at the edges of its row tiles and hidden chunks: one chunk, odd numbers of chunks, several tiles per CTA."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,dim,inner,dtype,ln", [(1, 128, 64, torch.bfloat16, True), (129, 64, 64, torch.float16, True), (128, 128, 192, torch.bfloat16, False),
                                                  (148 * 128 + 1, 128, 64, torch.bfloat16, True), (3 * 148 * 128 + 77, 64, 192, torch.bfloat16, True),
                                                  (2 * 148 * 128, 128, 320, torch.float16, True)])
def test_transition_chunks(M, dim, inner, dtype, ln):
    g = torch.Generator(device="cuda").manual_seed(M + inner)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, w1, w2, dy = r(M, dim).to(dtype), (r(dim, 2 * inner) / dim ** 0.5).to(dtype), (r(dim, inner) / inner ** 0.5).to(dtype), r(M, dim).to(dtype)
    lw, lb = ((1 + 0.1 * r(dim)).to(dtype), (0.1 * r(dim)).to(dtype)) if ln else (None, None)
    y, mean, rstd = mfb.transition_forward(x, lw, lb, w1, w2)
    assert _lib.last_path() == "tcgen05"
    f = lambda t: None if t is None else t.float()      # noqa: E731
    a = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        ref = orc.transition_fwd_bwd(f(x), f(lw), f(lb), f(w1), f(w2), f(dy))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = a
    assert_close_lowp(y, ref[0].cpu(), "y")
    if ln:
        got = mfb.transition_backward(dy, x, lw, lb, w1, w2, mean, rstd)
        for g_, r_, n in zip(got, ref[1:], ("dx", "d_ln_w", "d_ln_b", "dw1", "dw2")):
            assert float((g_.float() - r_).norm() / r_.norm()) < 2e-2, n
