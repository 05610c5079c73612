"""CPU: what autograd makes of the layer-level caller, with the op replaced by a plain convolution: derivatives of its gradients,
tangents and batched gradients of the bias, against the same layer written out in float64."""
import pytest
import torch
import torch.nn.functional as F

import tf_approximate_b200 as ax
from tf_approximate_b200 import layers, ops


def conv(x, w, strides, padding, dilations):
    """NHWC convolution with TensorFlow's padding."""
    sh, sw, dh, dw = strides[1], strides[2], dilations[1], dilations[2]
    x = x.permute(0, 3, 1, 2)
    if padding == "SAME":
        pads = [max((-(-size // s) - 1) * s + (k - 1) * d + 1 - size, 0)
                for size, s, k, d in ((x.shape[3], sw, w.shape[1], dw), (x.shape[2], sh, w.shape[0], dh))]
        x = F.pad(x, (pads[0] // 2, pads[0] - pads[0] // 2, pads[1] // 2, pads[1] - pads[1] // 2))
    return F.conv2d(x, w.permute(3, 2, 0, 1), stride=(sh, sw), dilation=(dh, dw)).permute(0, 2, 3, 1)


@pytest.fixture
def cpu_op(monkeypatch):
    def op(x, w, *_, strides, padding, dilations, bias=None, **__):
        y = conv(x, w, strides, padding, dilations).contiguous()
        if bias is not None and (bias.dtype != torch.float32 or tuple(bias.shape) != y.shape[3:]):
            raise ops.InvalidArgumentError("bias")         # (as the op does)
        return y if bias is None else y + bias
    monkeypatch.setattr(layers, "approx_conv2d_with_min_max_vars", op)
    monkeypatch.setattr(ops, "column_sums", lambda x: torch.from_numpy(x.detach().numpy().reshape(-1, x.shape[-1]).sum(0)))
    monkeypatch.setattr(ops, "tensor_range", lambda x, out: out.copy_(torch.stack([x.min(), x.max()])))
    monkeypatch.setattr(ops, "fake_quant_device_range", lambda x, r: layers.fake_quant_with_min_max_vars(x, r[0], r[1]))
    monkeypatch.setattr(layers.FakeApproxConv2D, "_own_buffers", lambda self, *a: (torch.empty(4), None))


def make(k=3, stride=1, padding="same", dilation=1, filters=5, hw=8, **kw):
    torch.manual_seed(k * 7 + stride + dilation)
    layer = ax.FakeApproxConv2D(4, filters, k, strides=stride, padding=padding, dilation_rate=dilation, mul_map_file="", **kw)
    if layer.bias is not None:
        with torch.no_grad():
            layer.bias.uniform_(-1, 1)
    return layer, torch.randn(2, hw, hw + 1, 4)


def in_float64(layer, x, kernel, bias):
    """The layer as autograd sees it: straight-through quantisation, the convolution, the bias."""
    def snap(t):
        q = layers.fake_quant_with_min_max_vars(t.detach().float(), t.detach().float().min(), t.detach().float().max())
        return t + (q.double() - t.detach())
    d = layer.dilation_rate
    y = conv(snap(x), snap(kernel), (1, *layer.strides, 1), layer.padding, (1, *d, 1))
    return y if bias is None else y + bias


def both(layer, x):
    """(fp32 leaves, float64 leaves) and the outputs of both."""
    leaves = [x.clone().requires_grad_(True), layer.kernel] + ([layer.bias] if layer.bias is not None else [])
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    return leaves, ref, layer(leaves[0]), in_float64(layer, *ref, *([None] if len(ref) == 2 else []))


# sums of at most a few thousand fp32 products of values about 1, differentiated twice
def close(a, b):
    return torch.allclose(a.double(), b, rtol=2e-5, atol=2e-5 * float(b.abs().max()))


SHAPES = [dict(), dict(stride=2), dict(stride=2, hw=9), dict(padding="valid"), dict(dilation=2), dict(k=1), dict(k=2), dict(k=5, padding="valid", stride=2)]


@pytest.mark.parametrize("kw", SHAPES, ids=str)
def test_gradients_and_their_derivatives(cpu_op, kw):
    layer, x = make(**kw)
    for of in ((2,), (0,), (1,), (0, 1, 2)):
        leaves, ref, y, y64 = both(layer, x)
        got = []
        for ls, out in ((leaves, y), (ref, y64)):
            loss = out.square().sum()
            grads = torch.autograd.grad(loss, [ls[i] for i in of], create_graph=True)
            (loss + sum((g * g).sum() for g in grads)).backward()
            got.append((grads, [t.grad for t in ls]))
            layer.zero_grad(set_to_none=True)
        assert all(close(a.detach(), b.detach()) for a, b in zip(got[0][0], got[1][0]))
        assert all(close(a, b) for a, b in zip(got[0][1], got[1][1])), of


def test_a_penalty_on_the_bias_gradient_alone(cpu_op):
    layer, x = make()
    y = layer(x)
    gb, = torch.autograd.grad(y.square().sum(), layer.bias, create_graph=True)
    assert gb.requires_grad
    gb.square().sum().backward()
    rows = y.numel() // y.shape[-1]
    assert close(layer.bias.grad, 4 * rows * gb.detach().double()) and layer.kernel.grad is not None


def test_tangent_of_the_bias(cpu_op):
    import torch.autograd.forward_ad as fwAD
    layer, x = make()
    bias, t = layer.bias.detach(), torch.randn(5)
    del layer.bias
    with fwAD.dual_level():
        layer.bias = fwAD.make_dual(bias, t)
        y, ty = fwAD.unpack_dual(layer(x))
        assert torch.equal(ty, t.expand(y.shape))


def test_batched_gradients(cpu_op):
    layer, x = make(filters=3, hw=4)
    leaves, ref, y, y64 = both(layer, x)
    v = torch.randn(6, *y.shape)
    got = torch.autograd.grad(y, leaves, v, is_grads_batched=True)
    for i in range(6):
        assert all(close(g[i], r) for g, r in zip(got, torch.autograd.grad(y64, ref, v[i].double(), retain_graph=True)))


@pytest.mark.parametrize("need", [(True, False, False), (False, True, False), (False, False, True), (False, True, True), (True, False, True)], ids=str)
@pytest.mark.parametrize("kw", [dict(), dict(stride=2)], ids=str)
def test_only_what_is_asked_for(cpu_op, kw, need):
    layer, x = make(**kw)
    x.requires_grad_(need[0])
    layer.kernel.requires_grad_(need[1])
    layer.bias.requires_grad_(need[2])
    y = layer(x)
    y.square().sum().backward()
    ref = [t.detach().double().requires_grad_(n) for t, n in zip((x, layer.kernel, layer.bias), need)]
    in_float64(layer, *ref).square().sum().backward()
    for t, r, n in zip((x, layer.kernel, layer.bias), ref, need):
        assert close(t.grad, r.grad) if n else t.grad is None


def test_no_bias(cpu_op):
    layer, x = make(use_bias=False)
    leaves, ref, y, y64 = both(layer, x)
    y.square().sum().backward()
    y64.square().sum().backward()
    assert all(close(a.grad, b.grad) for a, b in zip(leaves, ref))


def test_tangents_of_the_operands_are_refused(cpu_op):
    import torch.autograd.forward_ad as fwAD
    layer, x = make()
    with fwAD.dual_level(), pytest.raises(NotImplementedError):
        layer(fwAD.make_dual(x, torch.randn_like(x)))


@pytest.mark.parametrize("shape", [(1,), (), (1, 5), (9, 1), (8, 9, 5)], ids=str)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.bfloat16])
def test_biases_that_are_broadcast(cpu_op, shape, dtype):
    layer, x = make()
    bias = torch.randn(shape).to(dtype)
    layer.bias = torch.nn.Parameter(bias)
    y = layer(x)
    y.square().sum().backward()
    ref = [t.detach().double().requires_grad_(True) for t in (layer.kernel, bias)]
    y64 = in_float64(layer, x.double(), *ref)
    y64.square().sum().backward()
    assert close(y.detach(), y64.detach()) and close(layer.kernel.grad, ref[0].grad)
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2e-5      # the gradient has the bias's type
    assert torch.allclose(layer.bias.grad.double(), ref[1].grad, rtol=tol, atol=tol * float(ref[1].grad.abs().max()))
