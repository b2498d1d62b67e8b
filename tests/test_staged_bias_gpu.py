"""Forward with a pair bias that is staged in shared memory by the warps (fp32, or head sizes above 32): ragged last tiles,
one key, rows and keys just beyond a tile, a bias shared by the batch, padded rows, and a length whose mask rows leave no room."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,bias_dtype,L,D", [(torch.float16, torch.float32, 4, 64), (torch.bfloat16, torch.float32, 132, 64), (torch.float16, torch.float32, 260, 40),
                                                  (torch.bfloat16, torch.bfloat16, 264, 64), (torch.bfloat16, torch.float32, 388, 32), (torch.float16, torch.float16, 136, 48),
                                                  (torch.bfloat16, torch.float32, 2308, 64)])
@pytest.mark.parametrize("shared", [False, True])
def test_staged_bias(dtype, bias_dtype, L, D, shared):
    g = torch.Generator(device="cuda").manual_seed(L + D)
    B, N, H = (2, 2, 3) if L < 1000 else (1, 1, 1)
    q, k, v = (torch.randn(B, N, L, H, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    mask = torch.rand(B, N, 1, 1, L, device="cuda", generator=g) > 0.2
    mask[..., 0] = True
    bias = torch.randn(1 if shared else B, 1, H, L, L + 8, device="cuda", generator=g).to(bias_dtype)[..., :L].expand(B, 1, H, L, L)
    o, _ = mfb.evo_attention_forward(q, k, v, mask, bias)
    assert _lib.last_path() == "tcgen05"
    f = lambda t: t.float().cpu()      # noqa: E731
    assert_close_lowp(o, orc.evo_attention(f(q), f(k), f(v), mask.cpu(), f(bias)), f"o L={L} D={D}")
