"""The native entry points of the fused ops (csrc/torch/fused_ops.cpp) against the Python statement of the same ops, which runs when they
answer None: the same kernels in the same order, so results and gradients agree bit for bit, and calls outside their form behave alike."""
import contextlib
import math

import pytest
import torch

from oneflow_b200.framework import fused_ops as FO
from oneflow_b200.ops import kernels as K

pytestmark = pytest.mark.gpu
DEV, BF = "cuda", torch.bfloat16


@contextlib.contextmanager
def python_path():
    FO.op_trace = []
    try:
        yield
    finally:
        FO.op_trace = None


def _rand(*shape, grad=True, scale=0.5):
    return (torch.randn(*shape, device=DEV) * scale).to(BF).requires_grad_(grad)


def _run(f, tensors, dy, python):
    for t in tensors:
        t.grad = None
    with (python_path() if python else contextlib.nullcontext()):
        y = f(*tensors)
        if y.requires_grad:
            y.backward(dy(y) if callable(dy) else dy)
    return [y.detach()] + [t.grad for t in tensors]


def _compare(f, tensors, dy=torch.randn_like):
    torch.manual_seed(5)
    native = _run(f, tensors, dy, False)
    torch.manual_seed(5)
    python = _run(f, tensors, dy, True)
    for a, b in zip(native, python):
        assert (a is None) == (b is None)
        if a is not None:
            assert a.dtype == b.dtype and a.shape == b.shape and torch.equal(a, b)
    return native


def _misaligned(t):
    flat = torch.empty(t.numel() + 3, device=DEV, dtype=t.dtype)[3:]
    return flat.view(t.shape).copy_(t).detach().requires_grad_(t.requires_grad)


@pytest.mark.parametrize("act", [0, "gelu", "relu"])
@pytest.mark.parametrize("form", ["plain", "rows1", "batched", "strided_x", "misaligned_x", "wide_weight", "strided_weight", "no_bias",
                                  "residual", "strided_residual", "no_grad_x", "only_bias"])
def test_linear_forms(form, act):
    torch.manual_seed(1)
    x, w, b, r = _rand(37, 64), _rand(72, 64), _rand(72), None
    if form == "rows1":
        x = _rand(1, 64)
    elif form == "batched":
        x = _rand(3, 5, 64)
    elif form == "strided_x":
        x = _rand(64, 37).t().detach().requires_grad_()
    elif form == "misaligned_x":
        x = _misaligned(x)
    elif form == "wide_weight":
        w, b = _rand(3, 24, 64), _rand(3, 24)
    elif form == "strided_weight":
        w = _rand(72, 128)[:, :64].detach().requires_grad_()
    elif form == "no_bias":
        b = None
    elif form == "residual":
        r = _rand(37, 72)
    elif form == "strided_residual":
        r = _rand(37, 144)[:, :72].detach().requires_grad_()
    elif form == "no_grad_x":
        x = _rand(37, 64, grad=False)
    elif form == "only_bias":
        x, w = _rand(37, 64, grad=False), _rand(72, 64, grad=False)
    tensors = [t for t in (x, w, b, r) if t is not None]

    def f(*_):
        return FO.linear(x, w, b, act=act, residual=r)
    _compare(f, tensors)
    _compare(f, tensors, lambda y: torch.ones((), device=DEV, dtype=BF).expand(y.shape))     # a gradient without memory of its own
    with torch.no_grad():
        a = f()
        with python_path():
            assert torch.equal(a, f()) and not a.requires_grad


@pytest.mark.parametrize("act", ["gelu", "gelu_tanh", "relu", 0])
@pytest.mark.parametrize("frozen", [(), ("x",), ("x", "w1", "b1"), ("w1", "w2")])
def test_mlp_forms(act, frozen):
    torch.manual_seed(2)
    names = ("x", "w1", "b1", "w2", "b2", "r")
    t = dict(zip(names, (_rand(70, 64), _rand(136, 64, scale=0.1), _rand(136), _rand(64, 136, scale=0.1), _rand(64), _rand(70, 64))))
    for n in frozen:
        t[n].requires_grad_(False)

    def f(*_):
        return FO.mlp(t["x"], t["w1"], t["b1"], t["w2"], t["b2"], act=act, residual=t["r"])
    _compare(f, list(t.values()))
    # a second backward through the same graph gives the same gradients again, natively and in Python
    for python in (False, True):
        with (python_path() if python else contextlib.nullcontext()):
            y = f()
            wanted = [v for v in t.values() if v.requires_grad]
            g = torch.randn_like(y)
            one = torch.autograd.grad(y, wanted, g, retain_graph=True)
            two = torch.autograd.grad(y, wanted, g)
            for a, b in zip(one, two):
                # the folded activation gradient is rounded once, the separate one twice
                torch.testing.assert_close(a.float(), b.float(), rtol=2e-2, atol=3e-2 * float(a.float().pow(2).mean().sqrt()))


@pytest.mark.parametrize("shape", [(1, 8), (5, 3, 64), (513, 1024), (4, 4096)])
def test_layer_norm_forms(shape):
    torch.manual_seed(3)
    x, g, b = _rand(*shape), _rand(shape[-1]), _rand(shape[-1])
    _compare(lambda *_: FO.layer_norm(x, (shape[-1],), g, b), [x, g, b])
    g2, b2 = g.detach(), b.detach()
    _compare(lambda *_: FO.layer_norm(x, shape[-1], g2, b2, 1e-3), [x])
    xs = _rand(shape[-1], shape[0]).t().detach().requires_grad_()
    _compare(lambda *_: FO.layer_norm(xs, (shape[-1],), g, b), [xs, g, b])
    xm = _rand(*shape)
    with pytest.raises((RuntimeError, ValueError)):
        FO.layer_norm(xm, (shape[-1],), _misaligned(g), b)


@pytest.mark.parametrize("layout", ["token", "head", "packed", "unequal_rows"])
@pytest.mark.parametrize("Sq,Sk,H,Hk,D,causal", [(1, 1, 2, 2, 64, False), (65, 130, 4, 2, 128, True), (127, 127, 3, 3, 64, True)])
def test_attention_forms(layout, Sq, Sk, H, Hk, D, causal):
    import oneflow_b200 as flow
    torch.manual_seed(4)
    B = 2
    if layout == "head":
        q, k, v = _rand(B, H, Sq, D), _rand(B, Hk, Sk, D), _rand(B, Hk, Sk, D)
        leaves = [q, k, v]
        views = (lambda: (q, k, v))
    elif layout == "packed":
        q, kv = _rand(B, Sq, H, D), _rand(B, Sk, 2, Hk, D)
        leaves = [q, kv]
        views = (lambda: (q.transpose(1, 2), kv[:, :, 0].transpose(1, 2), kv[:, :, 1].transpose(1, 2)))
    elif layout == "unequal_rows":
        q, k, vv = _rand(B, Sq, H, D), _rand(B, Sk, Hk, D), _rand(B, Sk, 2 * Hk, D)
        leaves = [q, k, vv]
        views = (lambda: (q.transpose(1, 2), k.transpose(1, 2), vv[:, :, :Hk].transpose(1, 2)))
    else:
        q, k, v = _rand(B, Sq, H, D), _rand(B, Sk, Hk, D), _rand(B, Sk, Hk, D)
        leaves = [q, k, v]
        views = (lambda: tuple(t.transpose(1, 2) for t in (q, k, v)))

    def f(*_):
        return flow.nn.functional.scaled_dot_product_attention(*views(), is_causal=causal)
    if layout == "head" and Sq == 1:     # a single token whose strides are not those of a token row is refused
        for python in (False, True):
            with pytest.raises(ValueError):
                _run(f, leaves, torch.randn_like, python)
        return
    # dQ is summed by atomic additions in both paths: its last bits depend on their order
    torch.manual_seed(5)
    native = _run(f, leaves, torch.randn_like, False)
    torch.manual_seed(5)
    python = _run(f, leaves, torch.randn_like, True)
    assert torch.equal(native[0], python[0]) and f().stride() == native[0].stride()
    with python_path():
        assert f().stride() == native[0].stride()
    for a, b in zip(native[1:], python[1:]):
        torch.testing.assert_close(a.float(), b.float(), rtol=2.0 ** -7, atol=1e-5)
    with torch.no_grad():
        assert torch.equal(f(), native[0])


def test_packed_attention_and_cross_entropy():
    torch.manual_seed(6)
    qkv = _rand(3 * 77, 3, 128)

    def f(*_):
        return FO.fused_attention_qkv_packed(qkv, seq_len=77, head_size=64, causal=True)
    torch.manual_seed(5)
    a = _run(f, [qkv], torch.randn_like, False)
    torch.manual_seed(5)
    b = _run(f, [qkv], torch.randn_like, True)
    assert torch.equal(a[0], b[0])
    torch.testing.assert_close(a[1].float(), b[1].float(), rtol=2.0 ** -7, atol=1e-5)
    labels = torch.randint(0, 1000, (33,), device=DEV)
    labels[3] = -100
    x = _rand(33, 1000, scale=2.0)
    # the gradient takes the logits' storage, so every run has its own copy
    for lab in (labels, labels.int().long().repeat(2)[::2].contiguous(), labels.view(11, 3)):
        out = []
        for python in (False, True):
            leaf = x.detach().clone().requires_grad_()
            with (python_path() if python else contextlib.nullcontext()):
                loss = FO.sparse_softmax_cross_entropy(leaf * 1.0, lab)
                loss.mean().backward()
            out.append((loss.detach(), leaf.grad))
        assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def test_hooks_modes_and_transforms():
    """What stands between a call and its kernels is still seen: hooks on saved tensors, function modes, transforms, tangents."""
    torch.manual_seed(7)
    x, w, b = _rand(16, 64), _rand(64, 64), _rand(64)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t.cpu())[1], lambda t: t.to(DEV)):
        y = FO.linear(x, w, b)
    y.backward(torch.ones_like(y))
    assert seen and x.grad is not None
    ref = _run(lambda *_: FO.linear(x, w, b), [x, w, b], torch.ones_like, True)
    assert torch.equal(ref[1], x.grad)

    for transform in (lambda: torch.func.vmap(lambda t: FO.linear(t, w, b))(x.detach().view(2, 8, 64)),
                      lambda: torch.func.jvp(lambda t: FO.linear(t, w, b), (x.detach(),), (torch.ones_like(x),))):
        errors = []
        for python in (False, True):
            with (python_path() if python else contextlib.nullcontext()):
                with pytest.raises(Exception) as e:
                    transform()
                errors.append(type(e.value))
        assert errors[0] is errors[1]
    # a node downstream that hands back no gradient counts as zeros
    class _Nothing(torch.autograd.Function):
        @staticmethod
        def forward(ctx, t):
            return t.clone()

        @staticmethod
        def backward(ctx, d):
            return None
    _compare(lambda *_: _Nothing.apply(FO.linear(x, w, b)) + x, [x, w, b])
    # a result may be changed in place, an input that the backward needs may not
    q = _rand(1, 8, 2, 64)
    import oneflow_b200 as flow
    o = flow.nn.functional.scaled_dot_product_attention(*(q.transpose(1, 2),) * 3)
    o.mul_(2.0)
    h = x * 1.0
    y = FO.linear(h, w, b)
    h.mul_(2.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


def test_refusals_and_counts():
    x, w, b = _rand(16, 64), _rand(64, 64), _rand(64)
    for call, err in ((lambda: FO.linear(x, w, b.float()), TypeError), (lambda: FO.linear(x, _rand(64, 72), b), (ValueError, RuntimeError)),
                      (lambda: FO.linear(x, w, _misaligned(b)), TypeError)):
        with pytest.raises(err):
            call()
    n0 = K.launch_count
    FO.linear(x, w, b)
    assert K.launch_count == n0 + 1
    FO.layer_norm(x, (64,), b, b)
    assert K.launch_count == n0 + 2
    # on another stream, from another thread
    import threading
    out = []

    def work():
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.default_stream())
        with torch.cuda.stream(s):
            y = FO.mlp(x, w, b, w, b, act="gelu")
            y.sum().backward()
            out.append(y.detach())
        s.synchronize()
    t = threading.Thread(target=work)
    t.start()
    t.join()
    with python_path():
        assert torch.equal(out[0], FO.mlp(x, w, b, w, b, act="gelu").detach())
    assert math.isfinite(float(x.grad.float().sum()))
