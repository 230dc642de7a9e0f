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
