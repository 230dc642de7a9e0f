"""Performance cases of the JVP attention: what users of ``JVPAttn`` run, from the smallest call to the largest.

A case is one attention problem (B, H, N, D), a data type, a mask, the way it is called and whether gradients are taken:

  api    "dual_level"  ``JVPAttn.fwd_dual`` on dual tensors inside ``fwAD.dual_level()``
         "func_jvp"    ``JVPAttn.fwd_dual`` under ``torch.func.jvp``
         "dual"        ``JVPAttn.dual`` with explicit tangents
         "primal"      ``attention`` (``JVPAttn.fwd``), no tangents
  train  False: the outputs only. True: also the gradients of both outputs (primal: of the one output) with respect to
         every input, as the backward of a training step asks for them
  mask   "none", "causal", "bool" ((B,1,N,N), 90 % kept, diagonal kept), "block" (boolean, 128 x 128 blocks at 25 %, diagonal
         blocks kept), "padding" (boolean (B,1,1,N), a prefix of every sequence is kept), "additive" ((B,1,N,N), N(0,1) with
         10 % of the entries -inf, diagonal finite)
  verify whether the call checks the mask (``verify_attn_mask``, on by default)
  fused  q, k, v and their tangents are the views that a fused qkv projection gives, (B,N,3,H,D) permuted, and the upstream
         gradients arrive as transposed (B,N,H,D) tensors

Inputs, tangents and upstream gradients are N(0,1).
"""
import math

import torch
import torch.autograd.forward_ad as fwAD

from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
BYTES = {"bf16": 2, "fp16": 2, "fp32": 4}


def _case(name, B, H, N, D, dtype, mask="none", api="dual_level", train=True, verify=True, fused=False):
    c = dict(B=B, H=H, N=N, D=D, dtype=dtype, mask=mask, api=api, train=train, verify=verify, fused=fused)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the first row of the README benchmark: the shortest sequence the reference accepts, forward only; a call this
        # small is what its launches and its host work cost
        _case("jvp_n32_fp16", 2, 12, 32, 64, "fp16", train=False),
        # the CPU-reference configuration: a small fp32 problem with all six gradients (validation runs, small models)
        _case("train_n128_fp32", 2, 4, 128, 64, "fp32"),
        # a layer of the diffusion transformer of bench_dit.py: short sequences, many (batch, head) pairs, head dimension 72,
        # views of the fused projection, called under torch.func.jvp inside a training step
        _case("dit_layer_d72_bf16", 32, 16, 256, 72, "bf16", api="func_jvp", verify=False, fused=True),
        # forward-only JVP of a causal model in the middle of the README table (sampling, evaluation of a tangent)
        _case("jvp_causal_n1024_fp16", 2, 12, 1024, 64, "fp16", mask="causal", train=False),
        # ordinary training without tangents through the same module: causal, head dimension 128
        _case("primal_causal_d128_fp16", 4, 8, 1024, 128, "fp16", mask="causal", api="primal"),
        # masked training at the mask configurations' shape: a boolean mask with the default checks ...
        _case("bool_mask_n1024_bf16", 2, 8, 1024, 64, "bf16", mask="bool"),
        # ... and a general additive bias with excluded entries
        _case("additive_mask_n1024_bf16", 2, 8, 1024, 64, "bf16", mask="additive", api="dual", verify=False),
        # a batch of sequences of unequal length: nothing is a multiple of a tile, key padding mask, head dimension 96
        _case("padded_n777_d96_bf16", 5, 7, 777, 96, "bf16", mask="padding", api="func_jvp"),
        # the dense training configuration
        _case("train_n2048_d64_bf16", 4, 16, 2048, 64, "bf16"),
        # the fp32 row of the README benchmark, with its gradients
        _case("train_n2048_d64_fp32", 2, 12, 2048, 64, "fp32", api="dual"),
        # the widest head the reference takes
        _case("train_causal_d256_fp16", 2, 8, 1024, 256, "fp16", mask="causal"),
        # the headline: long causal sequences, head dimension 128
        _case("headline_n4096_d128_bf16", 8, 16, 4096, 128, "bf16", mask="causal"),
    ]


def _flops(c):
    fwd, bwd = (4, 10) if c["api"] == "primal" else (12, 30)
    kept = {"causal": 0.5, "padding": 0.75}.get(c["mask"], 1.0)
    if c["mask"] == "block":
        n = math.ceil(c["N"] / 128)
        kept = 0.25 + 0.75 / n
    return (fwd + (bwd if c["train"] else 0)) * c["B"] * c["H"] * c["N"] ** 2 * c["D"] * kept


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    dtype = rng.choice(["bf16", "bf16", "bf16", "fp16", "fp16", "fp32"])
    if dtype == "fp32":
        D = rng.choice([32, 64, 64, 64, 128])
    else:
        D = rng.choice([16, 32, 40, 64, 64, 64, 64, 72, 80, 96, 128, 128, 128, 256])
    N = _log(rng, 32, 4096)
    if rng.random() < 0.5:
        N = max(32, N // 32 * 32)
    B, H = _log(rng, 1, 32), rng.choice([1, 2, 3, 4, 6, 7, 8, 8, 12, 12, 16, 16])
    mask = rng.choice(["none", "none", "none", "causal", "causal", "causal", "bool", "block", "padding", "additive"])
    api = rng.choice(["dual_level", "dual_level", "func_jvp", "func_jvp", "dual", "primal"])
    c = _case(None, B, H, N, D, dtype, mask, api, train=rng.random() < 0.75, verify=rng.random() < 0.5,
              fused=rng.random() < 0.3)
    # no larger than the largest listed case of its kind (fp32 and heads above 128 are the costlier kind)
    like = "train_causal_d256_fp16" if D > 128 or (dtype == "fp32" and D > 64) else (
        "train_n2048_d64_fp32" if dtype == "fp32" else "headline_n4096_d128_bf16")
    most = _flops(next(x for x in listed() if x["name"] == like))
    while _flops(c) > most:
        if c["B"] > 1:
            c["B"] = c["B"] // 2
        elif c["H"] > 1:
            c["H"] = c["H"] // 2
        else:
            c["N"] = c["N"] * 3 // 4
    return c


def _mask(c, g):
    B, N, kind = c["B"], c["N"], c["mask"]
    if kind in ("none", "causal"):
        return None
    dev = "cuda"
    if kind == "padding":
        length = (torch.rand(B, device=dev, generator=g) * 0.5 + 0.5) * N
        return (torch.arange(N, device=dev)[None, :] < length[:, None]).view(B, 1, 1, N)
    if kind == "bool":
        m = torch.rand(B, 1, N, N, device=dev, generator=g) < 0.9
        m.diagonal(dim1=-2, dim2=-1).fill_(True)
        return m
    if kind == "block":
        nb = math.ceil(N / 128)
        m = torch.rand(B, 1, nb, nb, device=dev, generator=g) < 0.25
        m.diagonal(dim1=-2, dim2=-1).fill_(True)
        return m.repeat_interleave(128, -1).repeat_interleave(128, -2)[..., :N, :N].contiguous()
    m = torch.randn(B, 1, N, N, device=dev, generator=g)
    out = torch.rand(B, 1, N, N, device=dev, generator=g) < 0.1
    out.diagonal(dim1=-2, dim2=-1).fill_(False)
    return m.masked_fill(out, float("-inf")).to(DTYPES[c["dtype"]])


def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, H, N, D, dt = c["B"], c["H"], c["N"], c["D"], DTYPES[c["dtype"]]

    def normal(*shape):
        return torch.randn(*shape, device="cuda", generator=g).to(dt)

    if c["fused"]:
        ins = list(normal(B, N, 3, H, D).permute(2, 0, 3, 1, 4)) + list(normal(B, N, 3, H, D).permute(2, 0, 3, 1, 4))
        ups = [normal(B, N, H, D).transpose(1, 2) for _ in range(2)]
    else:
        ins = [normal(B, H, N, D) for _ in range(6)]
        ups = [normal(B, H, N, D) for _ in range(2)]
    if c["api"] == "primal":
        ins, ups = ins[:3], ups[:1]
    ins = [t.detach().requires_grad_(c["train"]) for t in ins]
    kw = dict(attn_mask=_mask(c, g), causal=c["mask"] == "causal", verify_attn_mask=c["verify"])
    return dict(api=c["api"], train=c["train"], ins=ins, ups=ups, kw=kw)


def run(state):
    ins, ups, kw = state["ins"], state["ups"], state["kw"]
    if state["api"] == "primal":
        outs = [attention(*ins, **kw)]
    elif state["api"] == "dual":
        outs = list(JVPAttn.dual(*ins, **kw))
    elif state["api"] == "func_jvp":
        outs = list(torch.func.jvp(lambda q, k, v: JVPAttn.fwd_dual(q, k, v, **kw), tuple(ins[:3]), tuple(ins[3:])))
    else:
        with fwAD.dual_level():
            q, k, v = (fwAD.make_dual(ins[i], ins[i + 3]) for i in range(3))
            out = fwAD.unpack_dual(JVPAttn.fwd_dual(q, k, v, **kw))
            outs = [out.primal, out.tangent]
    if not state["train"]:
        return outs
    grads = torch.autograd.grad(outs, ins, ups)
    return [o.detach() for o in outs] + list(grads)


def work(case):
    c = case
    n_in = 3 if c["api"] == "primal" else 6
    n_out = 1 if c["api"] == "primal" else 2
    # inputs and outputs of the forward; for the gradients also the upstream gradients and one gradient per input
    tensors = n_in + n_out + ((n_out + n_in) if c["train"] else 0)
    rows = c["B"] * c["H"] * c["N"]
    mask = {"bool": c["B"] * c["N"] ** 2, "block": c["B"] * c["N"] ** 2, "padding": c["B"] * c["N"],
            "additive": c["B"] * c["N"] ** 2 * BYTES[c["dtype"]]}.get(c["mask"], 0)
    return {"bytes": tensors * rows * c["D"] * BYTES[c["dtype"]] + mask, "flops": _flops(c)}


def tolerance(case):
    # bf16 operands carry 8 significant bits and fp16 ones 11, through two rounded products (scores, then probabilities times
    # values); fp32 is what products of split 16-bit operands accumulated in fp32 give
    return {"rel": {"bf16": 1e-2, "fp16": 2e-3, "fp32": 5e-5}[case["dtype"]]}
