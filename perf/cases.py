"""What a user of megafold_b200 has it do, as a list of timed cases over the package's public entry points.

A case is a dict of plain values.  ``kind`` says which entry point it goes through; the other fields are sizes, types and
options of that call.  The listed cases are the benchmark configurations of this repository (triangle attention at crop
384, single-representation attention, the pair Transition, the LayernormLinear around the attention, the Pairformer
block), the shapes of its tests and the sizes around them that training and inference meet: the tiny fp32 configuration,
inference on a chain whose length is no multiple of anything, the single track (hundreds of rows, 384 channels), head
size 64, mixed precision with fp32 parameters, operands that live in host memory.  ``draw`` gives cases of the same
ranges.  Values and distributions are those of ``megafold_b200.workloads``.
"""
import math

import torch

import megafold_b200 as mfb

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16}
SIZE = {"fp32": 4, "bf16": 2, "fp16": 2}


def listed():
    return [
        # the tiny fp32 configuration: a parity check or a debugging run, where launches and host work are everything
        dict(name="attn_tiny_fp32", kind="attention", B=1, N=64, L=64, H=4, D=32, dtype="fp32", bias="fp32", mask="pad", train=True),
        # triangle attention of a training step at crop 384, the benchmark's headline
        dict(name="attn_triangle_384", kind="attention", B=1, N=384, L=384, H=4, D=32, dtype="bf16", bias="bf16", mask="pad", train=True),
        # triangle attention when predicting one structure: no gradients, and a chain has the length it has
        dict(name="attn_triangle_infer_467", kind="attention", B=1, N=467, L=467, H=4, D=32, dtype="bf16", bias="bf16", mask="none", train=False),
        # single-representation attention with pair bias in training: one row, sixteen heads of 24
        dict(name="attn_single_768", kind="attention", B=2, N=1, L=768, H=16, D=24, dtype="bf16", bias="bf16", mask="drop", train=True),
        # the shape the reference's own attention benchmark runs: head size 64, fp32 pair bias
        dict(name="attn_heads64_384", kind="attention", B=4, N=1, L=384, H=32, D=64, dtype="fp16", bias="fp32", mask="none", train=True),
        # the q/k/v/gate projection of the pair representation at crop 384
        dict(name="lnl_pair_384", kind="lnl", M=147456, K=128, N=512, dtype="bf16", autocast=False, linear_bias=True, train=True),
        # the projection of the single representation, mixed precision: fp32 parameters and residual stream under autocast
        dict(name="lnl_single_autocast", kind="lnl", M=768, K=384, N=1536, dtype="fp32", autocast=True, linear_bias=True, train=True),
        # the pair Transition at crop 512
        dict(name="transition_pair_512", kind="transition", M=262144, dim=128, expansion=4, dtype="bf16", autocast=False, train=True),
        # the single track's Transition
        dict(name="transition_single_384", kind="transition", M=768, dim=384, expansion=4, dtype="bf16", autocast=False, train=True),
        # the MSA track's Transition (64 channels, a few hundred sequences of a ragged length) when predicting
        dict(name="transition_msa_infer", kind="transition", M=59661, dim=64, expansion=4, dtype="bf16", autocast=False, train=False),
        # attention whose operands stay in pinned host memory between the steps
        dict(name="attn_host_384", kind="host", B=1, N=384, L=384, H=4, D=32, dtype="bf16", bias="bf16", mask="pad"),
        # a whole Pairformer block, forward and backward, at the long crop
        dict(name="block_768", kind="block", L=768, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    """An integer of [lo, hi], spread over the logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["attention"] * 5 + ["lnl"] * 2 + ["transition"] * 3 + ["host", "block"])
    mask = rng.choice(["pad", "drop", "none"])
    if kind == "attention":
        sort = rng.choice(["tiny", "triangle", "triangle", "single", "heads64"])
        if sort == "tiny":
            L = _log_int(rng, 16, 128)
            return dict(kind=kind, B=1, N=_log_int(rng, 1, L), L=L, H=rng.choice([1, 2, 4, 8]), D=rng.choice([16, 24, 32]), dtype="fp32",
                        bias="fp32", mask=mask, train=True)
        dtype = rng.choice(["bf16", "bf16", "fp16"])
        if sort == "triangle":
            # crops are multiples of 8 or 16 in training; inference takes any length
            train = rng.random() < 0.6
            L = _log_int(rng, 48, 640)
            L = L // 8 * 8 if train and rng.random() < 0.6 else L
            return dict(kind=kind, B=1, N=L, L=L, H=4, D=32, dtype=dtype, bias=dtype, mask=mask, train=train)
        if sort == "single":
            L = _log_int(rng, 64, 1024)
            return dict(kind=kind, B=rng.choice([1, 2]), N=1, L=L, H=16, D=24, dtype=dtype, bias=dtype, mask=mask, train=rng.random() < 0.7)
        return dict(kind=kind, B=rng.choice([1, 2, 4]), N=1, L=_log_int(rng, 64, 768), H=rng.choice([8, 16, 32]), D=rng.choice([48, 64]),
                    dtype=dtype, bias=rng.choice([dtype, "fp32"]), mask=mask, train=rng.random() < 0.7)
    if kind == "lnl":
        K = rng.choice([64, 128, 128, 256, 384])
        autocast = rng.random() < 0.4
        return dict(kind=kind, M=_log_int(rng, 96, 200000 if K <= 128 else 20000), K=K, N=8 * _log_int(rng, 1, 128 if K <= 128 else 192),
                    dtype="fp32" if autocast else rng.choice(["bf16", "fp16"]), autocast=autocast, linear_bias=rng.random() < 0.5,
                    train=rng.random() < 0.7)
    if kind == "transition":
        dim = rng.choice([64, 128, 128, 256, 384])
        autocast = rng.random() < 0.3
        return dict(kind=kind, M=_log_int(rng, 96, 262144 if dim <= 128 else 20000), dim=dim, expansion=rng.choice([2, 4]),
                    dtype="fp32" if autocast else rng.choice(["bf16", "bf16", "fp16"]), autocast=autocast, train=rng.random() < 0.7)
    if kind == "host":
        L = _log_int(rng, 96, 384)
        dtype = rng.choice(["bf16", "fp16"])
        return dict(kind=kind, B=1, N=L, L=L, H=4, D=32, dtype=dtype, bias=dtype, mask=mask)
    return dict(kind=kind, L=_log_int(rng, 96, 640), dtype="bf16")


# ---------------------------------------------------------------------------------------------------------------- inputs
def _attention_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, N, L, H, D = (case[x] for x in "BNLHD")
    dt, bdt = DTYPES[case["dtype"]], DTYPES[case["bias"]]
    q, k, v, d_out = (torch.randn(B, N, L, H, D, device="cuda", generator=g).to(dt) for _ in range(4))
    bias = torch.randn(B, 1, H, L, L, device="cuda", generator=g).to(bdt)
    if case["mask"] == "drop":
        mask = torch.rand(B, N, 1, 1, L, device="cuda", generator=g) >= 0.1
        mask[..., 0] = True
    else:
        mask = torch.ones(B, N, 1, 1, L, dtype=torch.bool, device="cuda")
        if case["mask"] == "pad":
            mask[..., L - L // 12:] = False
    return q, k, v, d_out, mask, bias


def _module_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt = DTYPES[case["dtype"]]
    out_dt = torch.bfloat16 if case["autocast"] else dt
    randn = lambda *s: torch.randn(*s, device="cuda", generator=g)      # noqa: E731
    if case["kind"] == "lnl":
        M, K, N = case["M"], case["K"], case["N"]
        module = mfb.LayernormLinear(K, N, has_linear_bias=case["linear_bias"], device="cuda", dtype=dt)
        values = {"WEIGHT": 1 + 0.1 * randn(K), "BIAS": 0.1 * randn(K), "linear_weight": randn(K, N) / K ** 0.5, "linear_bias": 0.1 * randn(N)}
    else:
        M, K = case["M"], case["dim"]
        I = K * case["expansion"]
        N = K
        module = mfb.FusedTransition(K, expansion_factor=case["expansion"], device="cuda", dtype=dt)
        values = {"ff.0.WEIGHT": 1 + 0.1 * randn(K), "ff.0.BIAS": 0.1 * randn(K), "ff.0.linear_weight": randn(K, 2 * I) / K ** 0.5,
                  "ff.2.weight": randn(K, I) / I ** 0.5}
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.copy_(values[name])
    return module, randn(M, K).to(dt), randn(M, N).to(out_dt)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind in ("attention", "host"):
        q, k, v, d_out, mask, bias = _attention_inputs(case, seed)
        if kind == "host":
            state["args"] = [t.cpu().pin_memory() for t in (q, k, v, mask, bias, d_out)]
            return state
        if case["train"]:
            for t in (q, k, v, bias):
                t.requires_grad_(True)
        state.update(q=q, k=k, v=v, mask=mask, bias=bias, d_out=d_out)
    elif kind in ("lnl", "transition"):
        module, x, dy = _module_inputs(case, seed)
        if case["train"]:
            x.requires_grad_(True)
        state.update(module=module, x=x, dy=dy, leaves=[x, *module.parameters()])
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        L, dt = case["L"], DTYPES[case["dtype"]]
        torch.manual_seed(seed)
        block = mfb.PairformerBlock(device="cuda", dtype=dt)
        pair, single, d_pair, d_single = (torch.randn(*s, device="cuda", generator=g).to(dt) for s in ((L, L, 128), (L, 384)) * 2)
        mask = torch.arange(L, device="cuda") < L - math.ceil(0.05 * L)
        pair.requires_grad_(True)
        single.requires_grad_(True)
        state.update(block=block, pair=pair, single=single, mask=mask, d_out=[d_pair, d_single], leaves=[pair, single, *block.parameters()])
    return state


# ------------------------------------------------------------------------------------------------------------- one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "host":
        return dict(mfb.evoformer_fwd_bwd_host(*state["args"]))
    if kind == "attention":
        q, k, v, bias = state["q"], state["k"], state["v"], state["bias"]
        if not case["train"]:
            with torch.no_grad():
                return mfb.TritonEvoformer(q, k, v, state["mask"], bias)
        o = mfb.TritonEvoformer(q, k, v, state["mask"], bias)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v, bias), state["d_out"])]
    if kind == "block":
        pair, single = state["block"](state["pair"], state["single"], state["mask"])
        return [pair.detach(), single.detach(), *torch.autograd.grad([pair, single], state["leaves"], state["d_out"])]
    with torch.autocast("cuda", torch.bfloat16, enabled=case["autocast"]):
        if not case["train"]:
            with torch.no_grad():
                return state["module"](state["x"])
        y = state["module"](state["x"])
    return [y.detach(), *torch.autograd.grad(y, state["leaves"], state["dy"])]


# ------------------------------------------------------------------------------------------------- unavoidable work
def _attention_work(B, N, L, H, D, es, bs, train):
    """One input or output of the size of q each: q k v -> o, and d_o -> dq dk dv; the bias, and its gradient."""
    x, b = B * N * L * H * D, B * H * L * L
    return {"bytes": (8 if train else 4) * x * es + (2 if train else 1) * b * bs + B * N * L, "flops": (14 if train else 4) * x * L}


def _sum(*parts):
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def _lnl_work(M, K, N, es, ys, train, linear_bias=True):
    par = K * N + 2 * K + (N if linear_bias else 0)
    t = 2 if train else 1
    return {"bytes": t * (M * K * es + M * N * ys + par * es), "flops": (6 if train else 2) * M * K * N}


def _transition_work(M, dim, inner, es, ys, train):
    par = 3 * dim * inner + 2 * dim
    t = 2 if train else 1
    return {"bytes": t * (M * dim * es + M * dim * ys + par * es), "flops": (18 if train else 6) * M * dim * inner}


def work(case):
    kind = case["kind"]
    es = SIZE[case["dtype"]]
    if kind in ("attention", "host"):
        return _attention_work(case["B"], case["N"], case["L"], case["H"], case["D"], es, SIZE[case["bias"]], case.get("train", True))
    if kind == "lnl":
        return _lnl_work(case["M"], case["K"], case["N"], es, 2 if case["autocast"] else es, case["train"], case["linear_bias"])
    if kind == "transition":
        return _transition_work(case["M"], case["dim"], case["dim"] * case["expansion"], es, 2 if case["autocast"] else es, case["train"])
    # block: two triangle attentions and the pair Transition on [L, L, 128], attention with pair bias on [L, 384]; the pair
    # and single representations and their gradients cross memory once each way per operator
    L = case["L"]
    P = L * L
    tri = [_lnl_work(P, 128, 512, es, es, True), _attention_work(1, L, L, 4, 32, es, es, True), _lnl_work(P, 128, 4, es, es, True),
           {"bytes": 4 * P * 128 * es, "flops": 6 * P * 128 * 128}]
    single = [_lnl_work(L, 384, 1536, es, es, True), _attention_work(1, 1, L, 16, 24, es, es, True), _lnl_work(P, 128, 16, es, es, True),
              {"bytes": 4 * L * 384 * es, "flops": 6 * L * 384 * 384}]
    return _sum(*tri, *tri, _transition_work(P, 128, 512, es, es, True), *single)


def tolerance(case):
    # 16-bit operands of every product and 16-bit results; fp32 differs by the order of its sums
    if case["kind"] == "block":
        return {"rel": 2e-2}
    if case["dtype"] == "fp32" and not case.get("autocast"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 3e-3} if case["dtype"] == "fp16" else {"rel": 1e-2}
