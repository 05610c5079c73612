"""GPU: gradients of the layer-level caller, and their derivatives, against the same layer in float64: even and uneven padding, VALID, dilation,
1x1, gradients asked for one by one, no bias."""
import pytest

pytestmark = pytest.mark.gpu

# chains of at most 2^12 roundings of 2^-24 each, relative to the largest value of the result
TOL = 2.0 ** -12

SHAPES = [dict(), dict(stride=2), dict(padding="valid"), dict(dilation=2), dict(k=1), dict(k=2), dict(k=5, padding="valid", stride=2),
          dict(c=64, filters=64, hw=28)]


def make(k=3, stride=1, padding="same", dilation=1, c=8, filters=12, hw=12, use_bias=True):
    import torch
    import tf_approximate_b200 as ax
    torch.manual_seed(k + 10 * stride + dilation)
    layer = ax.FakeApproxConv2D(c, filters, k, strides=stride, padding=padding, dilation_rate=dilation, use_bias=use_bias, mul_map_file="").cuda()
    if use_bias:
        with torch.no_grad():
            layer.bias.uniform_(-1, 1)
    return layer, torch.randn(3, hw, hw + 1, c, device="cuda")


def in_float64(layer, x, kernel, bias):
    import torch
    import torch.nn.functional as F
    from tf_approximate_b200 import layers

    def snap(t):
        f = t.detach().float()
        return t + (layers.fake_quant_with_min_max_vars(f, f.min(), f.max()).double() - t.detach())
    x, w = snap(x).permute(0, 3, 1, 2), snap(kernel).permute(3, 2, 0, 1)
    if layer.padding == "SAME":
        need = [max((-(-size // s) - 1) * s + (k - 1) * d + 1 - size, 0) for size, s, k, d in
                zip(x.shape[:1:-1], layer.strides[::-1], w.shape[:1:-1], layer.dilation_rate[::-1])]
        x = F.pad(x, (need[0] // 2, need[0] - need[0] // 2, need[1] // 2, need[1] - need[1] // 2))
    y = F.conv2d(x, w, stride=layer.strides, dilation=layer.dilation_rate).permute(0, 2, 3, 1)
    return y if bias is None else y + bias


def close(a, b):
    return float((a.double() - b).abs().max()) <= TOL * float(b.abs().max())


@pytest.fixture
def fp32(built):
    import torch
    before = torch.backends.cudnn.allow_tf32
    torch.backends.cudnn.allow_tf32 = False
    yield
    torch.backends.cudnn.allow_tf32 = before


@pytest.mark.parametrize("use_bias", [True, False])
@pytest.mark.parametrize("kw", SHAPES, ids=str)
def test_gradients_and_their_derivatives(fp32, kw, use_bias):
    import torch
    layer, x = make(use_bias=use_bias, **kw)
    leaves = [x.requires_grad_(True), layer.kernel] + [layer.bias] * use_bias
    ref = [t.detach().double().requires_grad_(True) for t in leaves]
    y, y64 = layer(x), in_float64(layer, ref[0], ref[1], ref[2] if use_bias else None)
    assert close(y.detach(), y64.detach())
    v = torch.randn_like(y64)
    grads, grads64 = (torch.autograd.grad((out * out * v.to(out.dtype)).sum(), ls, create_graph=True) for out, ls in ((y, leaves), (y64, ref)))
    assert all(close(a.detach(), b.detach()) for a, b in zip(grads, grads64))
    # a penalty on the last gradient (of the bias where there is one), then on all of them
    for some, some64 in ((grads[-1:], grads64[-1:]), (grads, grads64)):
        second = torch.autograd.grad(sum(g.square().sum() for g in some), leaves, retain_graph=True)
        second64 = torch.autograd.grad(sum(g.square().sum() for g in some64), ref, retain_graph=True)
        assert all(close(a, b) for a, b in zip(second, second64))


@pytest.mark.parametrize("need", [(True, False, False), (False, True, False), (False, False, True)], ids=str)
@pytest.mark.parametrize("kw", [dict(), dict(stride=2)], ids=str)
def test_one_gradient_alone(fp32, kw, need):
    import torch
    layer, x = make(**kw)
    leaves = [x, layer.kernel, layer.bias]
    for t, n in zip(leaves, need):
        t.requires_grad_(n)
    ref = [t.detach().double().requires_grad_(n) for t, n in zip(leaves, need)]
    y = layer(x)
    v = torch.randn_like(y)
    y.backward(v)
    in_float64(layer, *ref).backward(v.double())
    for t, r, n in zip(leaves, ref, need):
        assert close(t.grad, r.grad) if n else t.grad is None


def test_batched_gradients_and_tangents_of_the_bias(fp32):
    import torch
    import torch.autograd.forward_ad as fwAD
    layer, x = make()
    y = layer(x)
    v = torch.randn(3, *y.shape, device="cuda")
    got = torch.autograd.grad(y, [layer.kernel, layer.bias], v, is_grads_batched=True, retain_graph=True)
    for i in range(3):
        assert all(close(g[i], r.double()) for g, r in zip(got, torch.autograd.grad(y, [layer.kernel, layer.bias], v[i], retain_graph=True)))
    bias, t = layer.bias.detach(), torch.randn(12, device="cuda")
    del layer.bias
    with fwAD.dual_level():
        layer.bias = fwAD.make_dual(bias, t)
        z, tz = fwAD.unpack_dual(layer(x))
        assert torch.equal(z, y) and torch.equal(tz, t.expand(y.shape))
