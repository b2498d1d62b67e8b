"""LayernormLinear and the Transition at row widths 192 to 384 with values at the ends of their ranges: what the CUDA-core
kernels give."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib

pytestmark = pytest.mark.gpu

FORCE = _lib.MF_FLAG_FORCE_SIMT


@pytest.mark.parametrize("what", ["nan value", "inf value", "nan gate", "large negative gate", "minus inf gate"])
def test_swiglu_of_non_finite_products(what):
    """Single hidden values that are not finite, or gates where exp(-gate) overflows: no result hides them."""
    M, dim, inner = 130, 256, 64
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x, lw, lb = r(M, dim).bfloat16(), torch.ones(dim, device="cuda").bfloat16(), torch.zeros(dim, device="cuda").bfloat16()
    w1, w2 = (r(dim, 2 * inner) / 16).bfloat16(), (r(dim, inner) / 8).bfloat16()
    lb[0] = 1.0
    x[:, 0] = x.float().mean(1).bfloat16()       # LN(x)[:, 0] is close to 1: column 0 of w1 is added to every row nearly as it is
    gate, value = inner + 3, 3
    w1[:, gate] = 0
    if what.startswith(("nan value", "inf value")):
        w1[0, gate], w1[0, value] = -100.0, float(what.split()[0])
    else:
        w1[0, gate] = {"nan": float("nan"), "large": -3e4, "minus": float("-inf")}[what.split()[0]]
    y, *_ = mfb.transition_forward(x, lw, lb, w1, w2)
    assert _lib.last_path() == "tcgen05"
    want, *_ = mfb.transition_forward(x, lw, lb, w1, w2, flags=FORCE)
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    if what != "large negative gate":
        assert bool(torch.isnan(want).all())
    ok = ~torch.isnan(want)
    torch.testing.assert_close(y[ok].float(), want[ok].float(), rtol=2e-2, atol=2e-2)
