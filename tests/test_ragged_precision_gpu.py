"""Attention at a length whose bias rows TMA cannot address: whichever kernel a call takes, the output is as close to the
64-bit result.  The general kernel (a call without scratch) takes probabilities relative to the running maximum and the bias
without a rounded factor; the kernel that the copied bias makes possible has to be no further off."""
import ctypes as C

import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from megafold_b200.evoattention import _fill_common
from oracle import pairformer_oracle as orc

pytestmark = pytest.mark.gpu


def rel(x, exact):
    return float((x.double() - exact).norm() / exact.norm())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,L,D", [(40, 131, 32), (30, 259, 32), (12, 467, 32), (30, 385, 24), (50, 99, 8)])
def test_ragged_forward_is_as_exact_as_the_general_kernel(N, L, D, dtype):
    H = 4
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = (torch.randn(1, N, L, H, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    bias = torch.randn(1, 1, H, L, L, device="cuda", generator=g).to(dtype)
    mask = torch.ones(1, N, 1, 1, L, dtype=torch.bool, device="cuda")
    exact = orc.evo_attention(q, k, v, mask, bias, torch.float64)
    o, _ = mfb.evo_attention_forward(q, k, v, mask, bias)
    a = _lib.EvoFwdArgs()
    _fill_common(a, q, k, v, mask, bias, 0)
    general, lse = torch.empty_like(o), torch.empty(1, N, H, L, device="cuda")
    a.o, a.lse = general.data_ptr(), lse.data_ptr()
    assert _lib.lib().mf_evo_fwd_workspace_bytes(C.byref(a)) > 0
    _lib.check(_lib.lib().mf_evo_fwd(C.byref(a), _lib.stream_ptr("cuda")), "mf_evo_fwd")
    # the two differ in how exponentials are formed and summed in fp32, 1e-6 of each: far below 1 % of a rounding to 16 bits
    assert rel(o, exact) <= 1.01 * rel(general, exact)

