"""The one-pass input side of the LayernormLinear backward at the edges of its row tiles, column slabs and resident weights."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,N,dtype,bias", [(1, 128, 8, torch.bfloat16, True), (127, 64, 64, torch.float16, True), (128, 128, 72, torch.bfloat16, False),
                                              (129, 128, 136, torch.float16, True), (300, 64, 1000, torch.bfloat16, True),
                                              (148 * 128 + 5, 128, 512, torch.bfloat16, True), (2 * 148 * 128 + 1, 64, 24, torch.bfloat16, True),
                                              (3 * 148 * 128, 128, 520, torch.float16, True), (260, 128, 2048, torch.bfloat16, True),
                                              (260, 128, 2056, torch.bfloat16, True)])
def test_lnl_backward_rows(M, K, N, dtype, bias):
    g = torch.Generator(device="cuda").manual_seed(M + N)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, w, dy = (1.5 * randn(M, K) + 0.3).to(dtype), (randn(K, N) / K ** 0.5).to(dtype), (randn(M, N) / N ** 0.5).to(dtype)
    ln_w, ln_b = (1 + 0.1 * randn(K)).to(dtype), (0.1 * randn(K)).to(dtype) if bias else None
    b = randn(N).to(dtype) if bias else None
    _, mean, rstd = mfb.layernorm_linear_forward(x, w, b, ln_w, ln_b)
    got = mfb.layernorm_linear_backward(dy, x, w, ln_w, ln_b, mean, rstd, bias)
    assert _lib.last_path() == "tcgen05"
    f = lambda t: None if t is None else t.float().cpu()      # noqa: E731
    _, dx, dlw, dlb, dw, db = orc.layernorm_linear_fwd_bwd(f(x), f(ln_w), f(ln_b), f(w), f(b), f(dy))
    for g_, r_, n in zip(got, (dx, dw, db, dlw, dlb), ("dx", "dw", "db", "d_ln_w", "d_ln_b")):
        if g_ is not None:
            assert_close_lowp(g_, r_, n, summed_over=1 if n == "dx" else M)
            assert float((g_.float().cpu() - r_).norm() / r_.norm()) < (6e-3 if n in ("dx", "dw") else 1e-3)
