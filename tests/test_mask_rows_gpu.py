"""Summary of boolean masks that do not depend on the query (key padding): the same bytes as for the expanded mask."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes,N,step", [("batch", 1, 1), ("head", 63, 1), ("both", 64, 1), ("none", 65, 1), ("batch", 256, 1), ("both", 777, 1),
                                           ("batch", 130, 3), ("head", 1100, 2)])
def test_padding_mask_summary(planes, N, step):
    from jvp_flash_attention_b200 import _lib
    B, H = 3, 2
    shape = {"none": (1, 1), "batch": (B, 1), "head": (1, H), "both": (B, H)}[planes]
    g = torch.Generator(device="cuda").manual_seed(N)
    wide = torch.rand(*shape, 1, N * step, device="cuda", generator=g) < 0.5
    m = wide[..., ::step]
    m[..., : min(N, 64)] = True                # a tile that needs no mask
    if N > 128:
        m[..., 64:128] = False                 # tiles with nothing kept
    full = m.expand(*shape, N, N).contiguous()
    got, want = (_lib.mask_summary(_lib.make_mask(x, B, H, N), x, B, H, N) for x in (m, full))
    p, n64 = shape[0] * shape[1], (N + 63) // 64
    fb, bb = (p * n64 * n64 + 255) // 256 * 256, p * n64 * n64 * 64 * 8
    assert torch.equal(got[: p * n64 * n64], want[: p * n64 * n64])
    assert torch.equal(got[fb: fb + 2 * bb], want[fb: fb + 2 * bb])
