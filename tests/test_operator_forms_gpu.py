"""The operators under torch's transforms and on unusual forms of their arguments: refused, or the plain call's values."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

import megafold_b200 as mfb

pytestmark = pytest.mark.gpu


def calls():
    """name -> (function of one tensor, that tensor)"""
    r = lambda *s: torch.randn(*s, device="cuda")      # noqa: E731
    k, bias, mask = r(1, 2, 24, 2, 16), r(1, 1, 2, 24, 24), torch.ones(1, 2, 1, 1, 24, dtype=torch.bool, device="cuda")
    lnl, tr, sw = mfb.LayernormLinear(32, 24, device="cuda"), mfb.FusedTransition(32, device="cuda"), mfb.FusedSwiGLU()
    return {"attention": (lambda q: mfb.TritonEvoformer(q, k, k, mask, bias), r(1, 2, 24, 2, 16)), "lnl": (lnl, r(6, 32)), "transition": (tr, r(6, 32)),
            "swiglu": (sw, r(6, 32))}


@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("name", ["attention", "lnl", "transition", "swiglu"])
def test_transforms_are_refused(name, grad):
    f, x = calls()[name]
    with torch.set_grad_enabled(grad):
        with fwAD.dual_level(), pytest.raises(RuntimeError):
            f(fwAD.make_dual(x, torch.ones_like(x)))
        with pytest.raises(RuntimeError):
            torch.func.vmap(f)(torch.stack([x, x]))
        f(x)


@pytest.mark.parametrize("amp", [False, True])
@pytest.mark.parametrize("grad", [True, False])
@pytest.mark.parametrize("name", ["attention", "lnl", "transition", "swiglu"])
def test_pending_negation(name, grad, amp):
    """An argument whose sign has not been written to memory yet, with and without a conversion on the way."""
    if name == "attention" and amp:
        pytest.skip("takes its types as they are")
    f, x = calls()[name]
    lazy = torch._neg_view(x)
    assert lazy.is_neg()
    with torch.set_grad_enabled(grad), torch.autocast("cuda", torch.bfloat16, enabled=amp):
        assert torch.equal(f(lazy), f(-x))


def test_backward_functions_refuse_gradients_of_another_size():
    """What the reshape of dy to the rows of x refused, and sizes that would be read out of range."""
    r = lambda *s: torch.randn(*s, device="cuda")      # noqa: E731
    x, w, lw, w2 = r(2, 3, 32), r(32, 64), r(32), r(32, 32)
    mean, rstd = r(6), r(6)
    f = lambda dy, m=mean, w=w: mfb.layernorm_linear_backward(dy, x, w, lw, None, m, rstd, False)      # noqa: E731
    g = lambda dy, m=mean, w=w: mfb.transition_backward(dy, x, lw, None, w, w2, m, rstd)      # noqa: E731
    for call, n in ((f, 64), (g, 32)):
        call(r(6, n))
        call(r(2, 3, n))
        for bad in (dict(dy=r(5, n)), dict(dy=r(6, n - 1)), dict(dy=r(6, n), m=r(5)), dict(dy=r(6, n), w=r(31, 64))):
            with pytest.raises(ValueError):
                call(**bad)
        with pytest.raises(RuntimeError):
            call(r(6, n).cpu())


@pytest.mark.parametrize("amp", [False, True])
@pytest.mark.parametrize("name", ["EvoformerAttention", "LayernormLinearFunction", "FusedSwiGLUFunction", "TransitionFunction"])
def test_subclass_of_an_operator_class(name, amp):
    """A subclass of an operator's autograd function that adds a step of its own on both ways."""
    import megafold_b200.fused_transition as ft
    cls = getattr(mfb, name, None) or getattr(ft, name)

    class Twice(cls):
        @staticmethod
        def forward(ctx, *args):
            return 2 * cls.forward(ctx, *args)

        @staticmethod
        def backward(ctx, g):
            return cls.backward(ctx, 2 * g)

    r = lambda *s: torch.randn(*s, device="cuda").requires_grad_(True)      # noqa: E731
    mask = torch.ones(1, 2, 1, 1, 24, dtype=torch.bool, device="cuda")
    args = {"EvoformerAttention": (r(1, 2, 24, 2, 16), r(1, 2, 24, 2, 16), r(1, 2, 24, 2, 16), mask, r(1, 1, 2, 24, 24)),
            "LayernormLinearFunction": (r(6, 32), r(32, 24), r(24), r(32), r(32), True, True), "FusedSwiGLUFunction": (r(6, 32),),
            "TransitionFunction": (r(6, 32), r(32), r(32), r(32, 64), r(32, 32))}[name]
    leaves = [a for a in args if torch.is_tensor(a) and a.requires_grad]
    with torch.autocast("cuda", torch.bfloat16, enabled=amp):
        want, got = 2 * cls.apply(*args), Twice.apply(*args)
    assert torch.equal(got, want)
    d = torch.randn_like(got)
    for a, b in zip(torch.autograd.grad(got, leaves, d), torch.autograd.grad(want, leaves, d)):
        # under autocast the parameter gradients of the subclass pass through bf16 on their way: 2^-9 of each value
        torch.testing.assert_close(a, b, rtol=4e-3 if amp else 1e-5, atol=1e-5)
