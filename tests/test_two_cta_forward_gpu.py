"""Head dimensions up to 64 with more blocks than SMs: the forward kernel that runs two CTAs per SM, at the edges of its tiles
(one row, one more and one less than a 64-key or 128-query tile), its padded columns, masks with dead tiles, and dropout."""
import pytest
import torch

from oracle.jvp_attention_oracle import closed_form_oracle, make_additive_mask, make_bool_mask, make_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available()
    return torch.device("cuda:0")


@pytest.mark.parametrize("dtype,D,N,kind", [
    (torch.float16, 64, 1, "none"), (torch.bfloat16, 64, 63, "causal"), (torch.float16, 64, 65, "bool"), (torch.bfloat16, 64, 129, "none"),
    (torch.float16, 64, 200, "causal"), (torch.bfloat16, 8, 127, "causal"), (torch.float16, 40, 130, "additive"),
    (torch.bfloat16, 56, 192, "bool"), (torch.bfloat16, 64, 193, "additive"), (torch.float16, 64, 256, "dead"),
])
def test_two_cta_forward(dev, dtype, D, N, kind):
    from jvp_flash_attention_b200 import _lib
    from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention
    B, H = 2, 120                                   # 240 units: above 1.5 blocks per SM for every N
    ts = make_inputs(B, H, N, D, dtype=dtype, seed=N + D, scale=0.5 if dtype == torch.bfloat16 else 1.0)
    mask = {"bool": lambda: make_bool_mask(B, N), "additive": lambda: make_additive_mask(B, N, dtype=dtype)}.get(kind, lambda: None)()
    if kind == "dead":                              # a dead row, a dead key tile and a dead 128-query tile
        mask = torch.ones(B, 1, N, N, dtype=torch.bool)
        mask[:, :, 5] = False
        mask[:, :, :, 64:128] = False
        mask[1, :, 128:256] = False
    kw = dict(attn_mask=None if mask is None else mask.to(dev), causal=kind == "causal")
    heads = [0, 1, 77, H - 1]                       # the oracle on some of the heads
    ref = closed_form_oracle(*[t[:, heads] for t in ts], attn_mask=mask, causal=kind == "causal")
    ins = [t.to(dev) for t in ts[:6]]
    O, tO = JVPAttn.dual(*ins, **kw)
    for n, t in (("O", O), ("tO", tO), ("O", attention(*ins[:3], **kw))):
        assert float((t[:, heads].double().cpu() - torch.from_numpy(ref[n])).abs().max()) <= 2e-2, n
    torch.cuda.synchronize()
    _lib.read_status(dev)


def test_two_cta_forward_dropout(dev):
    """The keep pattern depends on the unit, the query and the key alone: the first heads of a large call and the same heads in a
    call of their own (which the kernel with one CTA per SM runs) agree to the rounding of the outputs and of P, W."""
    from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention
    for dtype, tol in ((torch.bfloat16, 1e-2), (torch.float16, 2e-3)):
        ins = [t.to(dev) for t in make_inputs(1, 160, 200, 64, dtype=dtype, seed=5)[:6]]
        few = [t[:, :3].contiguous() for t in ins]
        kw = dict(dropout_p=0.3, dropout_seed=11)
        big, small = JVPAttn.dual(*ins, **kw), JVPAttn.dual(*few, **kw)
        for x, y in [*zip(big, small), (attention(*ins[:3], **kw), attention(*few[:3], **kw))]:
            d = (x[:, :3].double() - y.double()).norm() / y.double().norm()
            assert float(d) <= tol, float(d)
