"""Pair biases that TMA cannot address (odd row lengths, permuted views, fp32) through the copied-bias path of both directions."""
import ctypes as C

import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from megafold_b200.evoattention import _fill_common
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu
NAMES = ("o", "dq", "dk", "dv", "dbias")


def _case(B, L, H, dtype, bias_dtype, permuted, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v, d_o = (torch.randn(B, 2, L, H, 32, device="cuda", generator=g).to(dtype) for _ in range(4))
    mask = torch.rand(B, 2, 1, 1, L, device="cuda", generator=g) > 0.2
    mask[..., 0] = True
    bias = torch.randn(B, 1, L, L, H, device="cuda", generator=g).to(bias_dtype).permute(0, 1, 4, 2, 3)
    return q, k, v, d_o, mask, bias if permuted else bias.contiguous()


@pytest.mark.parametrize("dtype,bias_dtype", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16), (torch.bfloat16, torch.float32)])
@pytest.mark.parametrize("L", [1, 9, 127, 129, 251, 260])
@pytest.mark.parametrize("permuted", [False, True])
def test_copied_bias(L, dtype, bias_dtype, permuted):
    q, k, v, d_o, mask, bias = _case(2, L, 3, dtype, bias_dtype, permuted, L)
    o, lse = mfb.evo_attention_forward(q, k, v, mask, bias)
    got = (o,) + tuple(mfb.evo_attention_backward(d_o, q, k, v, mask, bias, o, lse))
    assert _lib.last_path() == "tcgen05"
    f = lambda t: t.float().cpu()      # noqa: E731
    ref = orc.evo_attention_fwd_bwd(f(q), f(k), f(v), mask.cpu(), f(bias), f(d_o))
    for g_, r_, n in zip(got, ref, NAMES):
        assert_close_lowp(g_, r_, f"{n} L={L}", summed_over=2 if n == "dbias" else 1)


def test_forward_without_scratch_takes_the_general_kernel():
    q, k, v, _, mask, bias = _case(1, 131, 2, torch.bfloat16, torch.bfloat16, False, 5)
    want, _ = mfb.evo_attention_forward(q, k, v, mask, bias)
    a = _lib.EvoFwdArgs()
    _fill_common(a, q, k, v, mask, bias, 0)
    o, lse = torch.empty_like(q), torch.empty(1, 2, 2, 131, device="cuda")
    a.o, a.lse = o.data_ptr(), lse.data_ptr()
    assert _lib.lib().mf_evo_fwd_workspace_bytes(C.byref(a)) > 0
    _lib.check(_lib.lib().mf_evo_fwd(C.byref(a), _lib.stream_ptr("cuda")), "mf_evo_fwd")
    assert_close_lowp(o, want.float().cpu(), "o without scratch")
