"""Additive masks and biases that hold -inf: keys without weight, from the first key tile on and in any kernel's tiles."""
import pytest
import torch

import megafold_b200 as mfb
from oracle import pairformer_oracle as orc
from util import assert_close_fp32, assert_close_lowp

pytestmark = pytest.mark.gpu


def inputs(N, L, H, D, dtype, bias_dtype):
    g = torch.Generator(device="cuda").manual_seed(L + D)
    q, k, v = (torch.randn(1, N, L, H, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    return q, k, v, torch.randn(1, 1, H, L, L, device="cuda", generator=g).to(bias_dtype)


@pytest.mark.parametrize("masked", [(0, 64), (0, 128), (0, 190), (64, 128)])
@pytest.mark.parametrize("D,dtype,bias_dtype", [(64, torch.bfloat16, torch.float32), (40, torch.float16, torch.float16), (32, torch.bfloat16, torch.float32),
                                                (32, torch.float32, torch.float32), (32, torch.bfloat16, torch.bfloat16)])
def test_additive_mask_of_minus_infinity(D, dtype, bias_dtype, masked):
    """A whole tile of keys at -inf before the first key with weight (tiles of 64 and 128 keys)."""
    N, L, H = 2, 200, 2
    q, k, v, bias = inputs(N, L, H, D, dtype, bias_dtype)
    mask = torch.zeros(1, N, 1, 1, L, device="cuda")
    mask[:, 1, ..., masked[0]:masked[1]] = float("-inf")
    want = orc.evo_attention(q, k, v, mask, bias)
    got, _ = mfb.evo_attention_forward(q, k, v, mask, bias)
    assert bool(torch.isfinite(got).all())
    (assert_close_fp32 if dtype == torch.float32 else assert_close_lowp)(got, want, f"o D={D} masked={masked}")


@pytest.mark.parametrize("L,D,dtype,bias_dtype", [(131, 32, torch.bfloat16, torch.bfloat16), (259, 32, torch.float16, torch.float16), (259, 24, torch.bfloat16, torch.bfloat16),
                                                  (136, 32, torch.float16, torch.float32), (136, 64, torch.bfloat16, torch.float32)])
def test_bias_of_minus_infinity_that_is_copied(L, D, dtype, bias_dtype):
    """-inf in a pair bias that reaches the tensor cores through a 16-bit copy (unaligned rows; fp32 in the backward pass), for
    single keys and for the whole first tile of some queries."""
    N, H = 3, 2
    q, k, v, bias = inputs(N, L, H, D, dtype, bias_dtype)
    g = torch.Generator(device="cuda").manual_seed(1)
    bias[torch.rand(bias.shape, device="cuda", generator=g) < 0.2] = float("-inf")
    bias[..., L - 1] = 0.5                       # every query keeps a key
    bias[:, :, 0, 5:20, :128] = float("-inf")
    mask = torch.ones(1, N, 1, 1, L, dtype=torch.bool, device="cuda")
    d_o = torch.randn(1, N, L, H, D, device="cuda", generator=g).to(dtype)
    want = orc.evo_attention_fwd_bwd(q, k, v, mask, bias, d_o)
    o, lse = mfb.evo_attention_forward(q, k, v, mask, bias)
    got = (o, *mfb.evo_attention_backward(d_o, q, k, v, mask, bias, o, lse))
    for name, x, y in zip(("o", "dq", "dk", "dv", "dbias"), got, want):
        assert bool(torch.isfinite(x).all()), name
        assert_close_lowp(x, y, f"{name} L={L}", summed_over=N if name == "dbias" else 1)
