"""Attention forward, head sizes up to 32: lengths around its blocks of 64 keys and pairs of blocks, numbers of work items around
the streams of a CTA and the CTAs of the GPU, maxima that grow from block to block, rows whose keys are all masked."""
import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from oracle import pairformer_oracle as orc
from util import assert_close_lowp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,L,H,D", [(1, 1, 1, 32), (2, 64, 1, 8), (1, 65, 3, 32), (37, 72, 4, 24), (149, 128, 1, 32), (3, 129, 1, 16), (5, 192, 30, 32),
                                     (2, 200, 2, 32), (1, 320, 5, 24), (4, 456, 1, 32),
                                     # six or more items a CTA: a stream goes from item to item, with an odd and an even number of blocks
                                     (1001, 64, 1, 32), (333, 72, 3, 8), (251, 192, 2, 32), (151, 320, 2, 24), (113, 384, 3, 32)])
@pytest.mark.parametrize("rising", [False, True])
def test_streams_and_blocks(dtype, N, L, H, D, rising):
    g = torch.Generator(device="cuda").manual_seed(N + L)
    q, k, v = (torch.randn(1, N, L, H, D, device="cuda", generator=g).to(dtype) for _ in range(3))
    mask = torch.rand(1, N, 1, 1, L, device="cuda", generator=g) > 0.2
    mask[..., 0] = True
    mask[:, N // 2] = N < 2                        # every key of one row masked, where there is another
    bias = torch.randn(1, 1, H, L, L, device="cuda", generator=g)
    if rising:                                     # the running maximum grows by some 14 in base 2 from pair to pair of blocks
        bias = bias + torch.arange(L, device="cuda") * 0.08
    bias = bias.to(dtype)
    o, lse = mfb.evo_attention_forward(q, k, v, mask, bias)
    assert _lib.last_path() == "tcgen05"
    f = lambda t: t.float().cpu()      # noqa: E731
    assert_close_lowp(o, orc.evo_attention(f(q), f(k), f(v), mask.cpu(), f(bias)), f"o N={N} L={L} H={H} D={D}")
    s = torch.einsum("bnihd,bnjhd->bnhij", f(q), f(k)) / D ** 0.5 + f(bias)
    want = torch.logsumexp(s.masked_fill(~mask.cpu(), -torch.finfo(torch.float32).max), -1)
    dead = ~mask.any(-1)[..., 0, 0].cpu()
    want[dead] = -torch.finfo(torch.float32).max   # how the backward recognises such a row
    # q k and the bias times a 16-bit sqrt(D) (off by at most 2.5e-4 of it), sums in fp32
    torch.testing.assert_close(lse.cpu(), want, rtol=1e-3, atol=1e-3 + 2.5e-4 * float(f(bias).abs().max()))
