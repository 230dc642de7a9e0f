"""The native host path on the GPU: the mask check that reads the mask's summary, and the tangent levels it takes."""
import pytest
import torch
import torch.autograd.forward_ad as fwAD

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev():
    assert torch.cuda.is_available()
    return torch.device("cuda:0")


@pytest.mark.parametrize("N", [33, 64, 130, 256])            # 33, 130: rows off the 16-byte grid (the generic summary kernel)
@pytest.mark.parametrize("shape", ["per head", "per batch", "keys only"])
def test_mask_check_verdicts(dev, N, shape):
    """One plane of several with nothing kept, or one NaN in the last row and column, is an AssertionError; the mask before
    that change is none; and the call after an error works."""
    from jvp_flash_attention_b200 import attention
    B, H = 3, 2
    q = torch.randn(B, H, N, 64, device=dev, dtype=torch.float16)
    full = {"per head": (B, H, N, N), "per batch": (B, 1, N, N), "keys only": (B, 1, 1, N)}[shape]
    keep = torch.zeros(full, dtype=torch.bool, device=dev)
    keep[..., -1, -1] = True                                  # a single kept entry per plane is enough
    attention(q, q, q, attn_mask=keep)
    keep[B - 1, -1] = False
    with pytest.raises(AssertionError, match="all False"):
        attention(q, q, q, attn_mask=keep)
    attention(q, q, q, attn_mask=keep, verify_attn_mask=False)
    for dtype in (torch.float16, torch.bfloat16, torch.float32):
        bias = torch.full(full, float("-inf"), dtype=dtype, device=dev)   # excluded everywhere: not an error for a float mask
        attention(q, q, q, attn_mask=bias)
        bias[..., -1, -1][B - 1] = float("nan")
        with pytest.raises(AssertionError, match="NaN"):
            attention(q, q, q, attn_mask=bias)


def test_tangents_that_cannot_be_taken_raise(dev):
    """``fwd`` and ``dual`` on dual tensors, and a second level of tangents, raise instead of dropping a tangent."""
    from jvp_flash_attention_b200.jvp_attention import JVPAttn, attention
    q, t = (torch.randn(1, 1, 64, 64, device=dev, dtype=torch.float16) for _ in range(2))
    with fwAD.dual_level():
        d = fwAD.make_dual(q, t)
        with pytest.raises(RuntimeError):
            attention(d, q, q)
        with pytest.raises(RuntimeError):
            JVPAttn.dual(d, q, q, t, t, t)
    inner = lambda x: torch.func.jvp(lambda y: JVPAttn.fwd_dual(y, q, q), (x,), (t,))[1]
    with pytest.raises(RuntimeError):
        torch.func.jvp(inner, (q,), (t,))


@pytest.mark.parametrize("dtype,D", [(torch.float16, 64), (torch.bfloat16, 128), (torch.float16, 256), (torch.bfloat16, 256), (torch.float32, 64)])
def test_first_cuda_work_of_a_thread(dev, dtype, D):
    """A call may be the first thing that a thread does on the GPU."""
    from concurrent.futures import ThreadPoolExecutor
    from jvp_flash_attention_b200 import attention
    q = torch.randn(1, 2, 128, D, device=dev, dtype=dtype)
    want = attention(q, q, q)
    with ThreadPoolExecutor(1) as thread:
        got = thread.submit(attention, q, q, q).result()
    assert torch.equal(got, want)


@pytest.mark.parametrize("forward,backward", [
    ((torch.float32, 64), (torch.float32, 64)), ((torch.float16, 256), (torch.bfloat16, 64)), ((torch.float32, 32), (torch.float16, 136)),
])
def test_two_threads_on_one_stream(dev, forward, backward):
    """Forward calls of one thread against backward calls of another, on the same stream and therefore with the same scratch
    (split operands, per-row statistics): each gives the bits it gives alone."""
    import threading
    from jvp_flash_attention_b200.jvp_attention import JVPAttn

    def inputs(dtype, D, seed):
        g = torch.Generator(device=dev).manual_seed(seed)
        return [torch.randn(2, 4, 256, D, device=dev, generator=g).to(dtype) for _ in range(8)]

    f = inputs(*forward, 1)
    b = inputs(*backward, 2)
    leaves = [t.requires_grad_() for t in b[:6]]
    outs = JVPAttn.dual(*leaves, causal=True)
    run_f = lambda: list(JVPAttn.dual(*f[:6]))
    run_b = lambda: list(torch.autograd.grad(outs, leaves, b[6:], retain_graph=True))
    want = [run_f(), run_b()]
    got, start = [None, None], threading.Barrier(2)

    def repeat(i, run):
        start.wait()
        got[i] = [run() for _ in range(60)]

    threads = [threading.Thread(target=repeat, args=(i, run)) for i, run in enumerate((run_f, run_b))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for w, results in zip(want, got):
        assert all(torch.equal(x, y) for r in results for x, y in zip(r, w))


def test_mask_check_inside_a_capture(dev):
    """The verdict is read on the host: refused while a graph is captured, without spoiling the capture or the calls after it;
    without the check a masked call can be captured."""
    from jvp_flash_attention_b200 import attention
    q = torch.randn(1, 2, 130, 64, device=dev, dtype=torch.float16)
    mask = torch.rand(1, 1, 130, 130, device=dev) < 0.9
    want = attention(q, q, q, attn_mask=mask)
    stream = torch.cuda.Stream(dev)
    stream.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(stream):
        attention(q, q, q, attn_mask=mask)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        with pytest.raises(RuntimeError):
            attention(q, q, q, attn_mask=mask)
        got = attention(q, q, q, attn_mask=mask, verify_attn_mask=False)
    assert torch.equal(attention(q, q, q, attn_mask=mask), want)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("own_streams", [False, True])
def test_mask_checks_on_two_threads(dev, own_streams):
    """Verdicts of masks that are checked at the same time reach the calls they belong to."""
    import threading
    from jvp_flash_attention_b200 import attention
    q = torch.randn(2, 2, 130, 64, device=dev, dtype=torch.float16)
    good = torch.rand(2, 1, 130, 130, device=dev) < 0.9
    bad = good.clone()
    bad[1] = False
    want = attention(q, q, q, attn_mask=good)
    torch.cuda.synchronize()
    wrong = []

    def repeat(first):
        with torch.cuda.stream(torch.cuda.Stream(dev) if own_streams else torch.cuda.current_stream(dev)):
            for i in range(50):
                try:
                    ok = (i + first) % 2 == 0 and torch.equal(attention(q, q, q, attn_mask=good), want)
                    if (i + first) % 2 == 1:
                        attention(q, q, q, attn_mask=bad)
                except AssertionError:
                    ok = (i + first) % 2 == 1
                if not ok:
                    wrong.append(i)

    threads = [threading.Thread(target=repeat, args=(f,)) for f in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
