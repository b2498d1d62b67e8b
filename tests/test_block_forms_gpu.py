"""The Pairformer block's native functions in the forms its composed operators take."""
import pytest
import torch

import megafold_b200 as mfb

pytestmark = pytest.mark.gpu


def make(L, dtype=torch.bfloat16, seed=3, **kw):
    torch.manual_seed(seed)
    block = mfb.PairformerBlock(device="cuda", dtype=dtype, **kw)
    pair, single, d_pair, d_single = (torch.randn(*s, device="cuda").to(dtype) for s in ((L, L, 128), (L, 384)) * 2)
    mask = torch.arange(L, device="cuda") < L - 2
    return block, pair.requires_grad_(True), single.requires_grad_(True), mask, [d_pair, d_single]


def go(block, pair, single, mask, d):
    out = block(pair, single, mask)
    return [*(o.detach() for o in out), *torch.autograd.grad(out, [pair, single, *block.parameters()], d)]


def close(got, want, block, tol=1e-2):
    """2e-3 is what a 16-bit rounding of each result leaves; the block chains about twenty of them."""
    names = ["x", "s", "d_pair", "d_single", *(n for n, _ in block.named_parameters())]
    for n, a, b in zip(names, got, want):
        assert a.shape == b.shape, n
        if not n.endswith("pair_ln_b"):      # 0 up to rounding errors (a softmax's logit gradients sum to 0): nothing to compare
            assert float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-6)) < tol, n


def test_strided_parameters():
    """Parameters held transposed or as slices of a wider array give what their contiguous copies give."""
    block, *rest = make(40)
    with torch.no_grad():
        for p in block.parameters():      # none of them as the constructor leaves them, so that a wrong order shows
            p.add_(0.1 * torch.randn_like(p))
    want = go(block, *rest)
    for p in block.parameters():
        p.data = p.data.t().contiguous().t() if p.dim() == 2 else torch.stack([p.data, -p.data], 1)[:, 0]
    assert not any(p.is_contiguous() for p in block.parameters()) and block._whole(rest[0], rest[1])
    close(go(block, *rest), want, block)


@pytest.mark.parametrize("dtype,amp", [(torch.bfloat16, torch.float16), (torch.float32, torch.bfloat16)], ids=["bf16-in-fp16", "fp32-in-bf16"])
def test_backward_inside_autocast(dtype, amp):
    """Forward outside, backward inside an autocast region of another type: the values of a backward outside."""
    block, pair, single, mask, d = make(40, dtype)
    out = block(pair, single, mask)
    assert block._whole(pair, single)
    values = [o.detach() for o in out]
    leaves = [pair, single, *block.parameters()]
    want = torch.autograd.grad(out, leaves, d, retain_graph=True)
    with torch.autocast("cuda", amp):
        got = torch.autograd.grad(out, leaves, d)
    assert all(a.dtype == b.dtype for a, b in zip(got, want))
    close([*values, *got], [*values, *want], block, 1e-2 if dtype != torch.float32 else 1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("heads,dim_head", [(48, 8), (33, 8), (32, 16)])
def test_many_heads(heads, dim_head, dtype):
    """More heads than one group of the pair-bias re-layout takes, against the composed operators."""
    from megafold_b200.pairformer_block import cuda_ops
    block, *rest = make(36, dtype, single_heads=heads, single_dim_head=dim_head, tri_heads=heads, tri_dim_head=dim_head)
    assert block._whole(rest[0], rest[1])
    got = go(block, *rest)
    block.native_ok, block.ops = False, cuda_ops()
    close(got, go(block, *rest), block, 1e-2 if dtype != torch.float32 else 1e-4)


def test_mask_of_any_shape_with_a_value_per_token():
    block, pair, single, mask, d = make(40)
    want = go(block, pair, single, mask, d)
    for m in (mask[None], mask.view(40, 1), torch.stack([mask, ~mask], 1)[:, 0]):
        assert torch.equal(block(pair, single, m)[0], want[0])


def test_injected_operators_are_used():
    """Operators set on a block that has already run with its own, and a block restored from a state without the newer fields."""
    from types import SimpleNamespace
    from megafold_b200.pairformer_block import cuda_ops
    block, pair, single, mask, _ = make(40)
    want = block(pair, single, mask)
    ops, seen = cuda_ops(), []
    block.ops = SimpleNamespace(lnl=ops.lnl, transition=ops.transition, attention=lambda *a: (seen.append(1), ops.attention(*a))[1])
    x, s = block(pair, single, mask)
    assert len(seen) == 3
    block.ops = None
    block.__dict__.pop("native_ok", None)
    assert torch.equal(block(pair, single, mask)[0], want[0]) and len(seen) == 3


def at_offset(t):
    """The same values at an address that is a multiple of 2 bytes only."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.detach().reshape(-1)
    return flat[1:].view(t.shape)


def test_inputs_at_any_address():
    block, pair, single, mask, d = make(40)
    want = go(block, pair, single, mask, d)
    got = go(block, at_offset(pair).requires_grad_(True), at_offset(single).requires_grad_(True), mask, [at_offset(t) for t in d])
    close(got, want, block)


@pytest.mark.parametrize("K", [128, 384])
def test_added_gradients_at_any_address(K):
    """mf_lnl_bwd_add with an addend that cannot be read in 16-byte pieces: its values, and the family of kernels it reports."""
    import ctypes as C
    from megafold_b200 import _lib
    M, N = 150, 64
    x, dy, add = (torch.randn(M, n, device="cuda").bfloat16() for n in (K, N, K))
    w, lw = torch.randn(K, N, device="cuda").bfloat16(), torch.ones(K, device="cuda").bfloat16()
    _, mean, rstd = mfb.layernorm_linear_forward(x, w, None, lw, None)
    got = {}
    for name, addend in (("tcgen05", add), ("simt", at_offset(add))):
        a = _lib.LnlBwdArgs()
        a.M, a.K, a.N, a.dtype = M, K, N, _lib.MF_BF16
        dx, dw, dlw = torch.empty_like(x), torch.empty(K, N, device="cuda"), torch.empty(K, device="cuda")
        a.x, a.ln_w, a.w, a.dy, a.mean, a.rstd = (t.data_ptr() for t in (x, lw, w, dy, mean, rstd))
        a.dx, a.dw, a.d_ln_w = dx.data_ptr(), dw.data_ptr(), dlw.data_ptr()
        ws = _lib.workspace(_lib.lib().mf_lnl_bwd_workspace_bytes(C.byref(a)), "cuda")
        a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
        _lib.check(_lib.lib().mf_lnl_bwd_add(C.byref(a), addend.data_ptr(), None, _lib.stream_ptr("cuda")), "mf_lnl_bwd_add")
        assert _lib.last_path() == name
        got[name] = dx, dw, dlw
    for a, b in zip(*got.values()):
        torch.testing.assert_close(a.float(), b.float(), rtol=2e-2, atol=2e-2 * float(b.float().abs().max()))
