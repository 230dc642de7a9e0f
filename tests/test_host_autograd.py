"""The autograd side of the native host path on the CPU: its operators with stand-ins for the kernels (the mathematics in plain
torch), so that what is recorded, saved and refused around the kernels is looked at without a GPU."""
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch
import torch.autograd.forward_ad as fwAD
import torch.nn.functional as F

B, H, N, D = 2, 2, 6, 8


def _scores(q, k, tq, tk, mask, causal, scale):
    s = q @ k.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool).triu(1), float("-inf"))
    if mask is not None:
        s = s.masked_fill(~mask, float("-inf")) if mask.dtype == torch.bool else s + mask
    ts = None if tq is None else (tq @ k.transpose(-1, -2) + q @ tk.transpose(-1, -2)) * scale
    return s.softmax(-1), ts


def _outputs(q, k, v, tq, tk, tv, mask, causal, scale):
    p, ts = _scores(q, k, tq, tk, mask, causal, scale)
    if tq is None:
        return [p @ v]
    w = p * (ts - (p * ts).sum(-1, keepdim=True))
    return [p @ v, w @ v + p @ tv]


def _fwd(q, k, v, tq, tk, tv, mask, causal, scale, dropout_p, seed, verify, tangents_taken):
    out = _outputs(q, k, v, tq, tk, tv, mask, causal, scale)
    out.append(torch.zeros(2, *q.shape[:3]))
    if mask is not None:
        out.append(torch.zeros(64, dtype=torch.uint8))
    return out


def _bwd(go, gto, q, k, v, tq, tk, tv, o, to, stats, mask, summary, causal, scale, dropout_p, seed):
    def gradients():
        ins = [t.detach().requires_grad_() for t in ((q, k, v) if gto is None else (q, k, v, tq, tk, tv))]
        outs = _outputs(*ins, *([None] * (6 - len(ins))), mask, causal, scale)
        ups = [torch.zeros_like(q) if go is None else go.detach(), None if gto is None else gto.detach()]
        return list(torch.autograd.grad(outs, ins, ups[:len(outs)]))

    with ThreadPoolExecutor(1) as thread:      # (a thread of its own: here, below autograd, nothing is recorded)
        return thread.submit(gradients).result()


@pytest.fixture(scope="module")
def ops(built_library):
    from jvp_flash_attention_b200 import _lib
    _lib.host()
    lib = torch.library.Library("jvpfa", "IMPL")
    # (below autograd: the kernels see plain tensors)
    lib.impl("fwd", lambda *a: [t.detach() for t in _fwd(*a)], "CPU")
    lib.impl("bwd", _bwd, "CPU")
    yield torch.ops.jvpfa
    lib._destroy()


def _call(ops, q, k, v, mask=None):
    return ops.attention(q, k, v, mask, False, D ** -0.5, 0.0, 0, False, True)


def _dual(ops, *ts, mask=None):
    return ops.attention_dual(*ts, mask, False, D ** -0.5, 0.0, 0, False)


def _inputs(n=6, requires_grad=True):
    g = torch.Generator().manual_seed(0)
    return [torch.randn(B, H, N, D, generator=g).requires_grad_(requires_grad) for _ in range(n)]


def _layer(ops, x, w):
    q, k, v = (F.layer_norm(x, (D,)) @ w[i] for i in range(3))
    y = x + _call(ops, q, k, v)
    return y + F.gelu(F.layer_norm(y, (D,)) @ w[3])


@pytest.mark.parametrize("tangent_of", ["input", "weights too"])
def test_backward_inside_the_dual_level(ops, tangent_of):
    """Nonlinear layers behind the attention hand it an upstream gradient that carries a tangent while the level is open: the
    gradients are those of a backward after the level, and of the same model without the operator."""
    x, t, gy = _inputs(3, requires_grad=False)
    g = torch.Generator().manual_seed(1)
    w = [(torch.randn(D, D, generator=g) / 3).requires_grad_() for _ in range(4)]
    tw = [torch.randn(D, D, generator=g) / 3 for _ in range(4)]

    def grads(inside, call_ops):
        with fwAD.dual_level():
            ws = [fwAD.make_dual(a, b) for a, b in zip(w, tw)] if tangent_of == "weights too" else w
            y, ty = fwAD.unpack_dual(_layer(call_ops, fwAD.make_dual(x, t), ws))
            loss = (y * gy).sum() + ty.square().sum()
            if inside:
                return torch.autograd.grad(loss, w)
        return torch.autograd.grad(loss, w)

    class Plain:
        @staticmethod
        def attention(q, k, v, mask, causal, scale, *_):
            (q, tq), (k, tk), (v, tv) = (fwAD.unpack_dual(a) for a in (q, k, v))
            return fwAD.make_dual(*_outputs(q, k, v, tq, tk, tv, mask, causal, scale))

    want = grads(False, Plain)
    for inside in (False, True):
        for a, b in zip(grads(inside, ops), want):
            torch.testing.assert_close(a, b, rtol=1e-4, atol=1e-5)


def test_tangent_of_an_upstream_gradient_is_not_dropped_silently(ops):
    """Under ``torch.func.jvp`` the tangent of the result is asked for: differentiating the backward raises."""
    q, k, v, go, tgo = _inputs(5, requires_grad=False)
    pull = lambda g: torch.func.vjp(lambda a: _call(ops, a, k, v), q)[1](g)[0]
    with pytest.raises(RuntimeError, match="not supported"):
        torch.func.jvp(pull, (go,), (tgo,))


def _recorded(ops, how, ts):
    """(outputs, tangent outputs) of a call whose q, k, v require a gradient, and nothing else does."""
    q, k, v, tq, tk, tv = ts
    if how == "plain":
        return [_call(ops, q, k, v)]
    if how == "dual":
        return list(_dual(ops, *ts))
    if how == "func_jvp":
        return list(torch.func.jvp(lambda *x: _call(ops, *x), (q, k, v), (tq, tk, tv)))
    with fwAD.dual_level():
        return list(fwAD.unpack_dual(_call(ops, *(fwAD.make_dual(p, t) for p, t in ((q, tq), (k, tk), (v, tv))))))


@pytest.mark.parametrize("how", ["plain", "dual", "func_jvp", "dual_level"])
def test_differentiating_the_backward_raises(ops, how):
    """``create_graph=True``: whichever way the call was recorded and with constant upstream gradients, the gradients are not
    constants; differentiating them raises."""
    ts = [t.requires_grad_(i < 3) for i, t in enumerate(_inputs(6, requires_grad=False))]
    outs = _recorded(ops, how, ts)
    grads = torch.autograd.grad(outs, ts[:3], [torch.ones_like(o) for o in outs], create_graph=True)
    assert all(g.requires_grad for g in grads)
    with pytest.raises(RuntimeError, match="differentiate twice"):
        grads[0].square().sum().backward()


@pytest.mark.parametrize("how", ["plain", "dual", "func_jvp", "dual_level"])
def test_inputs_changed_in_place_are_noticed(ops, how):
    """What the backward needs is saved with its version: an input that is changed before the backward raises."""
    leaves = [t.requires_grad_(i < 3) for i, t in enumerate(_inputs(6, requires_grad=False))]
    ts = [t * 1.0 if i < 3 else t for i, t in enumerate(leaves)]
    outs = _recorded(ops, how, ts)
    with torch.no_grad():
        ts[1].add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(outs, leaves[:3], [torch.ones_like(o) for o in outs])


@pytest.mark.parametrize("dual", [False, True])
def test_mask_summary_goes_through_saved_tensor_hooks(ops, dual):
    """Everything of the size of the mask that the call makes is offered to saved-tensor hooks (offloading, checkpointing), and
    the backward takes it from there."""
    ts = _inputs(6)
    mask = torch.ones(1, 1, N, N, dtype=torch.bool)
    kept = []

    def pack(t):
        kept.append(t)
        return len(kept) - 1

    with torch.autograd.graph.saved_tensors_hooks(pack, lambda i: kept[i]):
        outs = list(_dual(ops, *ts, mask=mask)) if dual else [_call(ops, *ts[:3], mask=mask)]
    assert sum(t.dtype == torch.uint8 for t in kept) == 1
    torch.autograd.grad(outs, ts[:3], [torch.ones_like(o) for o in outs])


@pytest.mark.parametrize("how", ["plain", "dual_level", "func_jvp", "dual"])
def test_tangent_of_the_mask_is_refused(ops, how):
    """The tangent of an additive mask is not part of what the kernels compute: refused instead of left out."""
    q, k, v, tq, tk, tv = _inputs(6, requires_grad=False)
    mask, tm = torch.zeros(1, 1, N, N), torch.ones(1, 1, N, N)
    with pytest.raises(RuntimeError, match="not supported"):
        if how == "func_jvp":
            torch.func.jvp(lambda a, m: _call(ops, a, k, v, mask=m), (q, mask), (tq, tm))
        with fwAD.dual_level():
            m = fwAD.make_dual(mask, tm)
            if how == "dual":
                _dual(ops, q, k, v, tq, tk, tv, mask=m)
            _call(ops, fwAD.make_dual(q, tq) if how == "dual_level" else q, k, v, mask=m)


def test_mask_that_requires_a_gradient(ops):
    """It gets none, and a loss on the outputs can be differentiated all the same when nothing else requires a gradient."""
    q, k, v, tq, tk, tv = _inputs(6, requires_grad=False)
    mask = torch.zeros(1, 1, N, N, requires_grad=True)
    for outs in ([_call(ops, q, k, v, mask=mask)], list(_dual(ops, q, k, v, tq, tk, tv, mask=mask))):
        sum(o.sum() for o in outs).backward()
        assert mask.grad is None
