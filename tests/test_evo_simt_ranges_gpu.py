"""CUDA-core attention at the edges of its 64 x 64 tiles, and d_pair_bias summed in one and in several ranges of rows."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_fp32

pytestmark = pytest.mark.gpu
NAMES = ("o", "dq", "dk", "dv", "dbias")


@pytest.mark.parametrize("B,N,L,H,D", [(1, 1, 1, 1, 1), (2, 7, 64, 1, 32), (1, 33, 65, 2, 31), (1, 4, 127, 1, 33), (1, 2, 129, 2, 65), (1, 5, 300, 9, 16)])
@pytest.mark.parametrize("strided", [False, True])
def test_tiles_and_ranges(B, N, L, H, D, strided):
    g = torch.Generator(device="cuda").manual_seed(L)
    pad = 3 if strided else 0            # rows that cannot be read four elements at a time
    q, k, v = (torch.randn(B, N, L, H, D + pad, device="cuda", generator=g)[..., pad:] for _ in range(3))
    d_o = torch.randn(B, N, L, H, D, device="cuda", generator=g)
    bias = torch.randn(B, 1, H, L, L, device="cuda", generator=g)
    mask = torch.rand(B, N, 1, 1, L, device="cuda", generator=g) > 0.2
    mask[..., 0] = True
    o, lse = mfb.evo_attention_forward(q, k, v, mask, bias)
    got = (o,) + tuple(mfb.evo_attention_backward(d_o, q, k, v, mask, bias, o, lse))
    assert _lib.last_path() == "simt"
    ref = orc.evo_attention_fwd_bwd(*(t.cpu() for t in (q, k, v, mask, bias, d_o)))
    for g_, r_, n in zip(got, ref, NAMES):
        assert_close_fp32(g_, r_, n)
