"""Attention with outputs and gradients in places of the caller's choosing, the block's element-wise pieces, and the block as
native functions against its composed form."""
import ctypes as C

import pytest
import torch

import megafold_b200 as mfb
from megafold_b200 import _lib
from megafold_b200.evoattention import _fill_common

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,L,D", [(3, 70, 32), (129, 8, 24), (2, 140, 64)])
def test_attention_layouts(N, L, D, dtype):
    """o and d_o with the row and token axes swapped, dq / dk / dv as slices of one merged gradient: the contiguous values."""
    H = 2
    g = torch.Generator(device="cuda").manual_seed(N + L)
    q, k, v, d_o = (torch.randn(1, N, L, H, D, device="cuda", generator=g).to(dtype) for _ in range(4))
    bias = torch.randn(1, 1, H, L, L, device="cuda", generator=g).to(dtype)
    mask = torch.rand(1, N, 1, 1, L, device="cuda", generator=g) > 0.2
    mask[..., 0] = True
    o, lse = mfb.evo_attention_forward(q, k, v, mask, bias)
    want = mfb.evo_attention_backward(d_o, q, k, v, mask, bias, o, lse)
    lib, st = _lib.lib(), _lib.stream_ptr("cuda")
    os_, merged = torch.zeros(L, N, H, D, device="cuda", dtype=dtype), torch.zeros(1, N, L, 4, H, D, device="cuda", dtype=dtype)
    d_os = d_o[0].transpose(0, 1).contiguous()
    lay = _lib.EvoLayout()
    tok = H * D
    for f in (lay.o, lay.d_o):
        f[:] = (N * L * tok, tok, N * tok)
    lay.d_qkv[:] = (4 * N * L * tok, 4 * L * tok, 4 * tok)
    a = _lib.EvoFwdArgs()
    _fill_common(a, q, k, v, mask, bias, 0)
    lse2 = torch.empty_like(lse)
    a.o, a.lse = os_.data_ptr(), lse2.data_ptr()
    need = lib.mf_evo_fwd_workspace_bytes(C.byref(a))
    ws = _lib.workspace(need, "cuda")
    _lib.check(lib.mf_evo_fwd_laid_out(C.byref(a), C.byref(lay), ws.data_ptr(), need, st), "forward")
    assert torch.equal(os_.transpose(0, 1), o[0]) and torch.equal(lse, lse2)
    b = _lib.EvoBwdArgs()
    _fill_common(b, q, k, v, mask, bias, 0)
    db = torch.empty_like(bias)
    b.dbias_dtype = _lib.dtype_code(dtype)
    b.o, b.d_o, b.lse, b.d_bias = os_.data_ptr(), d_os.data_ptr(), lse.data_ptr(), db.data_ptr()
    b.dq, b.dk, b.dv = (merged[:, :, :, i].data_ptr() for i in range(3))
    ws = _lib.workspace(lib.mf_evo_bwd_workspace_bytes(C.byref(b)), "cuda")
    b.workspace, b.workspace_bytes = ws.data_ptr(), ws.numel()
    _lib.check(lib.mf_evo_bwd_laid_out(C.byref(b), C.byref(lay), st), "backward")
    for name, x, y in zip(("dq", "dk", "dv", "dbias"), (*(merged[:, :, :, i] for i in range(3)), db), want):
        if name == "dq":      # its partial sums may meet in another order
            torch.testing.assert_close(x.float(), y.float(), rtol=2e-2, atol=1e-2, msg=name)
        else:
            assert torch.equal(x, y), name
    assert float(merged[:, :, :, 3].abs().max()) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,cols", [(1, 8), (300, 384), (4097, 128)])
def test_gate(rows, cols, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows)
    o, d = (torch.randn(rows, cols, device="cuda", generator=g).to(dtype) for _ in range(2))
    wide = (3 * torch.randn(rows, 2 * cols, device="cuda", generator=g)).to(dtype)
    gate = wide[:, cols:]
    of, gf = o.clone().requires_grad_(True), gate.clone().requires_grad_(True)
    ref = of * torch.sigmoid(gf)
    ref.backward(d)
    out, d_o, d_wide = torch.empty_like(o), torch.empty_like(o), torch.zeros_like(wide)
    lib, st, dt = _lib.lib(), _lib.stream_ptr("cuda"), _lib.dtype_code(dtype)
    _lib.check(lib.mf_gate_fwd(o.data_ptr(), gate.data_ptr(), 2 * cols, out.data_ptr(), rows, cols, dt, st), "gate")
    _lib.check(lib.mf_gate_bwd(d.data_ptr(), o.data_ptr(), gate.data_ptr(), 2 * cols, d_o.data_ptr(), d_wide[:, cols:].data_ptr(), 2 * cols, rows, cols, dt, st), "gate")
    for x, y in ((out, ref.detach()), (d_o, of.grad), (d_wide[:, cols:], gf.grad)):
        if dtype == torch.float32:
            torch.testing.assert_close(x, y, rtol=1e-5, atol=1e-6)
        else:           # the roundings of the composed operations (a sigmoid on the edge between two values may go either way)
            assert float((x != y).float().mean()) < 1e-3
    assert float(d_wide[:, :cols].abs().max()) == 0


@pytest.mark.parametrize("L,H,np_", [(1, 4, 8), (33, 4, 8), (96, 16, 16), (127, 3, 8), (33, 3, 5)])
@pytest.mark.parametrize("swap", [0, 1])
def test_bias_layout(L, H, np_, swap):
    rows = torch.randn(L * L, np_, device="cuda").bfloat16()
    planes = torch.empty(H, L, L, device="cuda", dtype=torch.bfloat16)
    lib, st = _lib.lib(), _lib.stream_ptr("cuda")
    _lib.check(lib.mf_bias_layout(rows.data_ptr(), planes.data_ptr(), L, np_, H, swap, 0, _lib.MF_BF16, st), "to planes")
    want = rows.view(L, L, np_)[..., :H].permute(2, 0, 1)
    assert torch.equal(planes, want.transpose(1, 2) if swap else want)
    back = torch.full_like(rows, 7)
    _lib.check(lib.mf_bias_layout(back.data_ptr(), planes.data_ptr(), L, np_, H, swap, 1, _lib.MF_BF16, st), "to rows")
    assert torch.equal(back[:, :H], rows[:, :H]) and float(back[:, H:].abs().max() if H < np_ else 0) == 0


@pytest.mark.parametrize("M,K,N,dtype", [(300, 128, 64, torch.bfloat16), (300, 384, 64, torch.bfloat16), (100, 128, 520, torch.float16), (50, 40, 24, torch.float32)])
def test_lnl_backward_with_added_gradients(M, K, N, dtype):
    g = torch.Generator(device="cuda").manual_seed(M)
    x, dy, add, add2 = (torch.randn(M, n, device="cuda", generator=g).to(dtype) for n in (K, N, K, K))
    w, lw = torch.randn(K, N, device="cuda", generator=g).to(dtype), torch.ones(K, device="cuda", dtype=dtype)
    _, mean, rstd = mfb.layernorm_linear_forward(x, w, None, lw, None)
    plain = mfb.layernorm_linear_backward(dy, x, w, lw, None, mean, rstd, False)[0]
    a = _lib.LnlBwdArgs()
    a.M, a.K, a.N, a.dtype = M, K, N, _lib.dtype_code(dtype)
    dx, dw, dlw = torch.empty_like(x), torch.empty(K, N, device="cuda"), torch.empty(K, device="cuda")
    a.x, a.ln_w, a.w, a.dy, a.mean, a.rstd = (t.data_ptr() for t in (x, lw, w, dy, mean, rstd))
    a.dx, a.dw, a.d_ln_w = dx.data_ptr(), dw.data_ptr(), dlw.data_ptr()
    ws = _lib.workspace(_lib.lib().mf_lnl_bwd_workspace_bytes(C.byref(a)), "cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    _lib.check(_lib.lib().mf_lnl_bwd_add(C.byref(a), add.data_ptr(), add2.data_ptr(), _lib.stream_ptr("cuda")), "mf_lnl_bwd_add")
    want = add2 + (add + plain)
    if dtype == torch.float32:
        torch.testing.assert_close(dx, want, rtol=1e-5, atol=1e-5)
    else:
        assert torch.equal(dx, want)


@pytest.mark.parametrize("L", [40, 129])
def test_block_native_equals_composed(L):
    from megafold_b200.pairformer_block import cuda_ops
    torch.manual_seed(L)
    block = mfb.PairformerBlock(device="cuda", dtype=torch.bfloat16)
    mask = torch.arange(L, device="cuda") < L - 3
    pair, single, dp, ds = (torch.randn(*s, device="cuda").bfloat16() for s in ((L, L, 128), (L, 384)) * 2)
    pair.requires_grad_(True)
    single.requires_grad_(True)

    def go():
        x, s = block(pair, single, mask)
        return [x, s, *torch.autograd.grad([x, s], [pair, single, *block.parameters()], [dp, ds])]

    assert block._whole(pair, single)
    got = go()
    block.native_ok, block.ops = False, cuda_ops()
    want = go()
    names = ["x", "s", "d_pair", "d_single", *(n for n, _ in block.named_parameters())]
    for n, a, b in zip(names, got, want):
        if n.endswith("pair_ln_b"):      # 0 up to rounding errors (a softmax's logit gradients sum to 0): nothing to compare
            continue
        assert float((a.float() - b.float()).norm() / b.float().norm().clamp_min(1e-6)) < 1e-2, n
