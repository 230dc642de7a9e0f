"""Head dimensions 136 to 256 in fp16 / bf16 on the tensor cores, at the edges of their tiles: 64-column slabs (partly or wholly
beyond the head dimension), the two column halves of the forward (80 | 56 at 136), 128-row and 64-column tiles, one tile only."""
import pytest
import torch

from oracle.jvp_attention_oracle import GRAD_NAMES, closed_form_oracle, make_additive_mask, make_bool_mask, make_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available()
    return torch.device("cuda:0")


@pytest.mark.parametrize("dtype,D,N,kind", [
    (torch.float16, 136, 65, "none"), (torch.float16, 136, 200, "causal"), (torch.bfloat16, 144, 129, "causal"),
    (torch.float16, 192, 1, "none"), (torch.bfloat16, 192, 330, "none"), (torch.float16, 200, 128, "bool"),
    (torch.float16, 256, 63, "causal"), (torch.bfloat16, 256, 448, "causal"), (torch.float16, 256, 321, "bool"),
    (torch.bfloat16, 256, 192, "additive"), (torch.float16, 248, 300, "additive"),
])
def test_wide_heads(dev, dtype, D, N, kind):
    from jvp_flash_attention_b200 import _lib
    from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention
    # bf16 at half the scale: 8-bit mantissas cannot hold gradients of magnitude 8 to within 2e-2 (as in test_parity_gpu.py)
    ts = make_inputs(2, 3, N, D, dtype=dtype, seed=N + D, scale=0.5 if dtype == torch.bfloat16 else 1.0)
    mask = {"bool": lambda: make_bool_mask(2, N), "additive": lambda: make_additive_mask(2, N, dtype=dtype)}.get(kind, lambda: None)()
    kw = dict(attn_mask=None if mask is None else mask.to(dev), causal=kind == "causal")
    ref = closed_form_oracle(*ts, attn_mask=mask, causal=kind == "causal")
    # every input as a view of a wider tensor: read in place through its strides
    leaves = [torch.cat([t, t], dim=-1).to(dev)[..., :D].detach().requires_grad_(True) for t in ts[:6]]
    O, tO = JVPAttn.dual(*leaves, **kw)
    grads = torch.autograd.grad([O, tO], leaves, [ts[6].to(dev), ts[7].to(dev)])
    got = dict(zip(("O", "tO") + GRAD_NAMES, (O.detach(), tO.detach(), *grads)))
    worst = {n: float((t.double().cpu() - torch.from_numpy(ref[n])).abs().max()) for n, t in got.items()}
    assert max(worst.values()) <= 2e-2, worst
    # primal only
    z = torch.zeros_like(ts[0])
    ref = closed_form_oracle(*ts[:3], z, z, z, ts[6], z, attn_mask=mask, causal=kind == "causal")
    o = attention(*leaves[:3], **kw)
    g = torch.autograd.grad(o, leaves[:3], ts[6].to(dev))
    for n, t in zip(("O", "dq", "dk", "dv"), (o.detach(), *g)):
        assert float((t.double().cpu() - torch.from_numpy(ref[n])).abs().max()) <= 2e-2, n
    torch.cuda.synchronize()
    _lib.read_status(dev)


@pytest.mark.parametrize("dtype,B,H,N,D,causal,dual", [
    (torch.bfloat16, 2, 40, 257, 256, True, True), (torch.float16, 3, 25, 130, 136, False, True),
    (torch.bfloat16, 2, 2, 2500, 192, False, True), (torch.float16, 2, 2, 2500, 256, False, False),
])
def test_many_units_equal_few(dev, dtype, B, H, N, D, causal, dual):
    """A backward with more blocks than SMs, or with 40 column tiles a block (the value families then run through their score
    buffers many times), against the same (batch, head) units in calls of their own: the same bits."""
    from jvp_flash_attention_b200 import _lib
    g = torch.Generator(device=dev).manual_seed(N + D)
    ts = [torch.randn(B, H, N, D, device=dev, generator=g).to(dtype) for _ in range(8)]

    def run(b, h):
        q, k, v, tq, tk, tv, go, gto = (t[b, h].contiguous() for t in ts)
        if not dual:
            tq = tk = tv = gto = None
        mask = _lib.make_mask(None, *q.shape[:3])
        o, to, lse2, mu = _lib.fwd(q, k, v, tq, tk, tv, mask, None, causal, D ** -0.5)
        return _lib.bwd(q, k, v, tq, tk, tv, o, to, lse2, mu, go, gto, mask, None, causal, D ** -0.5)

    whole = run(slice(None), slice(None))
    assert all(t.isfinite().all() for t in whole)
    for h in (0, H // 2, H - 1):
        part = run(slice(B - 1, B), slice(h, h + 1))
        assert all(torch.equal(a[B - 1, h], b[0, 0]) for a, b in zip(whole, part)), h
    torch.cuda.synchronize()
    _lib.read_status(dev)


# What is left when everything but the outputs is held in 32 bits: the rounding of the outputs, in the 2-norm 2^-p sqrt(0.541 / 12)
# for numbers of p bits whose significands are spread as 1/x (2.07e-4 in fp16, 1.66e-3 in bf16), and the rounding of O inside
# rowsum(O gO). One more rounding to 16 bits on the way (of the probabilities, of the score gradients) makes it sqrt(2) of that.
ROUNDING = {torch.float16: 2.0 ** -10 * (0.541 / 12) ** 0.5, torch.bfloat16: 2.0 ** -7 * (0.541 / 12) ** 0.5}


@pytest.mark.parametrize("dtype,D,N,kind,scale", [
    (torch.float16, 136, 320, "none", 1.0), (torch.float16, 256, 130, "bool", 1.0), (torch.bfloat16, 136, 130, "none", 1.0),
    (torch.bfloat16, 256, 320, "bool", 1.0), (torch.float16, 256, 320, "none", 6e3), (torch.bfloat16, 200, 192, "none", 1e6),
])
def test_errors_are_those_of_the_rounded_outputs(dev, dtype, D, N, kind, scale):
    """Also with upstream gradients of a magnitude whose score gradients do not fit the inputs' type."""
    from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention
    ts = make_inputs(2, 3, N, D, dtype=dtype, seed=N + D)
    ts = [*ts[:6], *((t.float() * scale).to(dtype) for t in ts[6:])]
    mask = make_bool_mask(2, N) if kind == "bool" else None
    kw = dict(attn_mask=None if mask is None else mask.to(dev))
    z = torch.zeros_like(ts[0])
    for primal in (False, True):
        leaves = [t.to(dev).requires_grad_(True) for t in ts[:3 if primal else 6]]
        outs = [attention(*leaves, **kw)] if primal else list(JVPAttn.dual(*leaves, **kw))
        grads = torch.autograd.grad(outs, leaves, [t.to(dev) for t in ts[6:6 + len(outs)]])
        ref = closed_form_oracle(*ts[:3], *((z, z, z, ts[6], z) if primal else ts[3:]), attn_mask=mask)
        names = ("O", "dq", "dk", "dv") if primal else ("O", "tO") + GRAD_NAMES
        for n, t in zip(names, (*outs, *grads)):
            want = torch.from_numpy(ref[n])
            err = float((t.detach().double().cpu() - want).norm() / want.norm())
            assert err <= 1.2 * ROUNDING[dtype], (primal, n, err)


def test_fp16_batches_beyond_the_workspace_bound(dev):
    """fp16 calls whose split operands exceed the bound of the workspace run in groups of batches (the forward four and one, the
    backward one by one): the same bits as a batch in a call of its own."""
    from jvp_flash_attention_b200 import _lib
    B, H, N, D = 5, 32, 4096, 256
    g = torch.Generator(device=dev).manual_seed(3)
    ts = [torch.randn(B, H, N, D, device=dev, generator=g, dtype=torch.float16) for _ in range(8)]

    def run(b):
        q, k, v, tq, tk, tv, go, gto = (t[b] for t in ts)
        mask = _lib.make_mask(None, *q.shape[:3])
        o, to, lse2, mu = _lib.fwd(q, k, v, tq, tk, tv, mask, None, True, D ** -0.5)
        return (o, to, lse2, mu) + _lib.bwd(q, k, v, tq, tk, tv, o, to, lse2, mu, go, gto, mask, None, True, D ** -0.5)

    whole = run(slice(0, B))
    for b in (0, B - 1):
        assert all(torch.equal(x[b], y[0]) for x, y in zip(whole, run(slice(b, b + 1))))
    torch.cuda.synchronize()
    _lib.read_status(dev)


def test_fp16_without_room_for_the_split_operands(dev):
    """The smallest workspace is still taken: contiguous fp16 inputs then run on the CUDA cores, as far from the outputs of the
    tensor cores as two roundings to fp16 are."""
    import ctypes as C
    from jvp_flash_attention_b200 import _lib
    B, H, N, D = 1, 2, 130, 136
    q, k, v, tq, tk, tv = (torch.randn(B, H, N, D, device=dev, dtype=torch.float16) for _ in range(6))
    mask = _lib.make_mask(None, B, H, N)
    want = _lib.fwd(q, k, v, tq, tk, tv, mask, None, False, D ** -0.5)
    a = _lib.FwdArgs()
    a.B, a.H, a.N, a.D, a.dtype, a.causal, a.sm_scale, a.mask = B, H, N, D, _lib.F16, 0, D ** -0.5, mask
    a.q, a.k, a.v, a.tq, a.tk, a.tv = (t.data_ptr() for t in (q, k, v, tq, tk, tv))
    got = [torch.empty_like(t) for t in want]
    a.o, a.to, a.lse2, a.mu = (t.data_ptr() for t in got)
    assert _lib.lib().jvpfa_fwd_workspace_bytes(C.byref(a)) > 256
    ws = torch.zeros(256, dtype=torch.uint8, device=dev)
    a.workspace, a.workspace_bytes = ws.data_ptr(), 256
    _lib.check(_lib.lib().jvpfa_fwd(C.byref(a), _lib.stream_ptr(dev)))
    for x, y in zip(got, want):
        assert float((x.double() - y.double()).norm() / y.double().norm()) <= 2 ** 0.5 * 1.2 * ROUNDING[torch.float16]
