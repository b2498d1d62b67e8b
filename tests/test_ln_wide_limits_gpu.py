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


@pytest.mark.parametrize("K", [192, 256, 384])
def test_normalised_values_beyond_fp16(K):
    """|LN(x)| up to 80000 in fp16, where the products with small weights are ordinary numbers."""
    M, N = 140, 72
    g = torch.Generator(device="cuda").manual_seed(K)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    x = (0.01 * r(M, K)).half()
    x[torch.arange(M), torch.randint(K, (M,), device="cuda", generator=g)] = 30.0      # one element of sqrt(K) standard deviations
    gain = torch.full((K,), 80000 / K ** 0.5, device="cuda").half()
    w = (1e-3 * r(K, N)).half()
    y, *_ = mfb.layernorm_linear_forward(x, w, None, gain, None)
    assert _lib.last_path() == "tcgen05"
    want, *_ = mfb.layernorm_linear_forward(x, w, None, gain, None, flags=FORCE)
    assert bool(torch.isfinite(want).all())
    torch.testing.assert_close(y, want, rtol=2e-3, atol=2e-3 * float(want.abs().max()))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_nan_rows_stay_nan(dtype):
    """A row of x with a NaN or an infinity is NaN in the result, the rows beside it are not touched."""
    r = torch.randn(140, 256, device="cuda").to(dtype)
    r[3, 7], r[131, 0] = float("nan"), float("inf")
    w, gain = (torch.randn(256, 64, device="cuda") / 16).to(dtype), torch.ones(256, device="cuda").to(dtype)
    y, *_ = mfb.layernorm_linear_forward(r, w, None, gain, None)
    assert bool(torch.isnan(y[[3, 131]]).all()) and bool(torch.isfinite(y[[i for i in range(140) if i not in (3, 131)]]).all())


@pytest.mark.parametrize("offset,path", [(0, "tcgen05"), (2, "simt"), (8, "simt"), (16, "tcgen05")])
def test_transition_workspace_at_any_address(offset, path):
    """mf_transition_fwd with a workspace that is aligned for its elements only."""
    import ctypes as C
    M, dim, inner = 130, 256, 64
    x, w1, w2 = (torch.randn(*s, device="cuda").bfloat16() for s in ((M, dim), (dim, 2 * inner), (dim, inner)))
    lw = torch.ones(dim, device="cuda").bfloat16()
    want, mean, rstd = mfb.transition_forward(x, lw, None, w1, w2)
    y = torch.empty_like(x)
    a = _lib.TransitionFwdArgs()
    a.M, a.dim, a.inner, a.dtype, a.eps = M, dim, inner, _lib.MF_BF16, 1e-5
    a.x, a.ln_w, a.w1, a.w2, a.y, a.mean, a.rstd = (t.data_ptr() for t in (x, lw, w1, w2, y, mean, rstd))
    need = _lib.lib().mf_transition_fwd_workspace_bytes(C.byref(a))
    ws = torch.empty(need + 64, dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr() + offset, need
    assert _lib.lib().mf_transition_fwd_workspace_bytes(C.byref(a)) == need
    _lib.check(_lib.lib().mf_transition_fwd(C.byref(a), _lib.stream_ptr("cuda")), "mf_transition_fwd")
    assert _lib.last_path() == path
    torch.testing.assert_close(y.float(), want.float(), rtol=2e-2, atol=2e-2 * float(want.float().abs().max()))
