"""Forward of LayernormLinear and Transition for rows of 192 to 384 elements: edges of row tiles, column blocks and CTAs."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu


def _rand(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return lambda *s: torch.randn(*s, device="cuda", generator=g)


def _check(y, ref, name):
    assert _lib.last_path() == "tcgen05"
    assert_close_lowp(y, ref, name)
    # only the result is rounded to 16 bit: half a unit in the last place is at most 2^-9 (bf16) or 2^-12 (fp16)
    rel = float((y.float().cpu() - ref).norm() / ref.norm())
    assert rel < (2e-3 if y.dtype == torch.bfloat16 else 2.6e-4), (name, rel)


@pytest.mark.parametrize("M,K,N,dtype,bias", [(1, 384, 8, torch.bfloat16, True), (128, 192, 64, torch.float16, False), (129, 320, 72, torch.bfloat16, True),
                                              (768, 384, 1536, torch.bfloat16, True), (700, 256, 1000, torch.float16, True), (5000, 384, 1528, torch.bfloat16, False)])
def test_lnl_forward(M, K, N, dtype, bias):
    r = _rand(M + N)
    x, w = (2 * r(M, K) + 0.5).to(dtype), (r(K, N) / K ** 0.5).to(dtype)
    lw, lb, b = (1 + 0.1 * r(K)).to(dtype), (0.1 * r(K)).to(dtype) if bias else None, r(N).to(dtype) if bias else None
    y, mean, rstd = mfb.layernorm_linear_forward(x, w, b, lw, lb)
    f = lambda t: None if t is None else t.float().cpu()      # noqa: E731
    _check(y, orc.layernorm_linear(f(x), f(lw), f(lb), f(w), f(b)), "y")
    torch.testing.assert_close(mean.cpu(), f(x).mean(1), rtol=1e-5, atol=1e-5)
    torch.testing.assert_close(rstd.cpu(), (f(x).var(1, unbiased=False) + 1e-5).rsqrt(), rtol=1e-4, atol=1e-5)


@pytest.mark.parametrize("M,dim,inner,dtype", [(1, 384, 32, torch.bfloat16), (128, 256, 96, torch.float16), (769, 384, 1536, torch.bfloat16),
                                               (3000, 192, 768, torch.bfloat16)])
def test_transition_forward(M, dim, inner, dtype):
    r = _rand(M + inner)
    x, w1, w2 = r(M, dim).to(dtype), (4 * r(dim, 2 * inner) / dim ** 0.5).to(dtype), (r(dim, inner) / inner ** 0.5).to(dtype)
    lw, lb = (1 + 0.1 * r(dim)).to(dtype), (0.1 * r(dim)).to(dtype)
    y, _, _ = mfb.transition_forward(x, lw, lb, w1, w2)
    f = lambda t: t.float().cpu()      # noqa: E731
    ref = orc.transition(f(x), f(lw), f(lb), f(w1), f(w2))
    assert _lib.last_path() == "tcgen05"
    assert float((f(y) - ref).abs().max()) < 2e-2 * float(ref.abs().max())
    assert float((f(y) - ref).norm() / ref.norm()) < (2.8e-3 if dtype == torch.bfloat16 else 3.6e-4)      # the gated product is rounded too
