"""Attention backward with several work items a CTA: their numbers step through heads, rows and batch elements, and dQ leaves the
accumulators of one item while the next is under way."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,L,H,D", [(3, 37, 136, 3, 32), (3, 101, 128, 2, 32), (1, 75, 384, 4, 24), (2, 83, 520, 1, 32), (1, 149, 768, 1, 32),
                                       (2, 51, 200, 3, 64)])
def test_many_items_a_cta(B, N, L, H, D):
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v, d_o = (torch.randn(B, N, L, H, D, device="cuda", generator=g).bfloat16() for _ in range(4))
    mask = torch.rand(B, N, 1, 1, L, device="cuda", generator=g) > 0.2
    mask[..., 0] = True
    bias = torch.randn(B, 1, H, L, L, device="cuda", generator=g).bfloat16()
    o, lse = mfb.evo_attention_forward(q, k, v, mask, bias)
    got = mfb.evo_attention_backward(d_o, q, k, v, mask, bias, o, lse)
    assert _lib.last_path() == "tcgen05"
    ref = orc.evo_attention_fwd_bwd(q.float(), k.float(), v.float(), mask, bias.float(), d_o.float())[1:]
    for g_, r_, n in zip(got, ref, ("dq", "dk", "dv", "dbias")):
        assert_close_lowp(g_, r_, f"{n} B={B} N={N} L={L}", summed_over=N if n == "dbias" else 1)
    # one CTA a (b, n, h) and dQ on chip: every product is there, so every call gives the same bits
    for _ in range(3):
        for a, b in zip(got, mfb.evo_attention_backward(d_o, q, k, v, mask, bias, o, lse)):
            assert torch.equal(a, b)
