"""All families of a backward in one launch: the same bits as with one launch per family (the form that records events between
them), where the families have fewer blocks than SMs, share a last wave, or end in a ragged row tile. (Head dimensions above 128
have one form only: test_wide_heads_gpu.py compares its many blocks with calls of few.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,B,H,N,D,causal,dual", [
    (torch.bfloat16, 1, 1, 1, 64, False, True), (torch.float16, 2, 5, 129, 64, True, True), (torch.bfloat16, 1, 3, 200, 72, False, True),
    (torch.float16, 3, 50, 130, 128, True, True), (torch.bfloat16, 1, 149, 65, 128, False, False), (torch.float16, 1, 75, 257, 40, True, False),
    (torch.float32, 1, 2, 130, 64, True, True), (torch.float32, 2, 40, 192, 32, False, False),
])
def test_one_launch_equals_one_per_family(dtype, B, H, N, D, causal, dual):
    from jvp_flash_attention_b200 import _lib
    g = torch.Generator(device="cuda").manual_seed(N + D)
    q, k, v, tq, tk, tv, go, gto = (torch.randn(B, H, N, D, device="cuda", generator=g).to(dtype) for _ in range(8))
    if not dual:
        tq = tk = tv = gto = None
    mask = _lib.make_mask(None, B, H, N)
    o, to, lse2, mu = _lib.fwd(q, k, v, tq, tk, tv, mask, None, causal, D ** -0.5)
    events = [torch.cuda.Event(enable_timing=True) for _ in range(5)]
    for e in events:
        e.record()
    one, many = (_lib.bwd(q, k, v, tq, tk, tv, o, to, lse2, mu, go, gto, mask, None, causal, D ** -0.5, marks=m) for m in (None, events))
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) and a.isfinite().all() for a, b in zip(one, many))
