"""Transition backward (dim = 128) where its tiles, chunks and teams change hands: one chunk, odd numbers of chunks, a tile
more than the grid has blocks, ragged last tiles, more rows than one range."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,inner,dtype,shift", [(1, 32, torch.bfloat16, True), (128, 96, torch.float16, False), (33, 64, torch.bfloat16, True),
                                                 (3 * 148 * 128 + 77, 32, torch.bfloat16, True), (2 * 148 * 128 + 1, 160, torch.float16, True),
                                                 (262144 + 129, 64, torch.bfloat16, True)])
def test_transition_bwd_chunks(M, inner, dtype, shift):
    g = torch.Generator(device="cuda").manual_seed(M + inner)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, w1, w2, dy = r(M, 128).to(dtype), (r(128, 2 * inner) / 128 ** 0.5).to(dtype), (r(128, inner) / inner ** 0.5).to(dtype), r(M, 128).to(dtype)
    lw, lb = (1 + 0.1 * r(128)).to(dtype), (0.1 * r(128)).to(dtype) if shift else None
    xf = x.float()
    mean, rstd = xf.mean(1), (xf.var(1, unbiased=False) + 1e-5).rsqrt()
    got = mfb.transition_backward(dy, x, lw, lb, w1, w2, mean, rstd)
    assert _lib.last_path() == "tcgen05"
    f = lambda t: None if t is None else t.float()      # noqa: E731
    a = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = False
    try:
        ref = orc.transition_fwd_bwd(f(x), f(lw), f(lb) if shift else torch.zeros(128, device="cuda"), f(w1), f(w2), f(dy))
    finally:
        torch.backends.cuda.matmul.allow_tf32 = a
    for g_, r_, n in zip(got, ref[1:], ("dx", "d_ln_w", "d_ln_b", "dw1", "dw2")):
        if g_ is not None:
            assert float((g_.float() - r_).norm() / r_.norm()) < 2e-2, n
