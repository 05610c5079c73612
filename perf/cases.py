"""The framework's work as its users have it do it, with the sizes that performance is measured at.

Every case is one pass through a public entry point: a table convolution (dense, depthwise, quantised, or in the
reference's order of additions), the layer-level caller with its backward pass, or a whole network.  Sizes are those
of the ResNet-50, ResNet-20 and depthwise-separable workloads in `workloads.py` and of the repository's tests; `draw`
gives more cases of the same ranges."""
import numpy as np
import torch

import tf_approximate_b200 as ax
from tf_approximate_b200 import workloads

DEVICE = torch.device("cuda", 0)


# ---------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------
def conv(kind, n, h, w, c, k, cout, stride=1, table="truncated", padding="SAME", dilation=1, signed=False, input_relu=False,
         bias=False, residual=False, relu=False):
    return {"kind": kind, "n": n, "h": h, "w": w, "c": c, "k": k, "cout": cout, "stride": stride, "table": table, "padding": padding,
            "dilation": dilation, "signed": signed, "input_relu": input_relu, "bias": bias, "residual": residual, "relu": relu}


def listed():
    return [
        # the reference's single-layer example: eight CIFAR-sized images, exact products; a call is mostly latency
        dict(conv("dense", 8, 32, 32, 16, 3, 32, table="exact", signed=True), name="cifar_conv_exact_b8"),
        # one image in the last stage of ResNet-50: few pixels, many channels, long K (interactive use)
        dict(conv("dense", 1, 7, 7, 512, 3, 512, input_relu=True), name="image_conv_7x7_512"),
        # the 3x3 layer of the first stage at the benchmark's batch, a multiplier without any structure
        dict(conv("dense", 256, 56, 56, 64, 3, 64, table="noisy"), name="conv_56x56_64_noisy"),
        # the expanding 1x1 layer of a bottleneck with the shortcut and the ReLU that follow it (short K, large output)
        dict(conv("dense", 64, 56, 56, 64, 1, 256, input_relu=True, residual=True, relu=True), name="expand_1x1_residual"),
        # the 3x3 layer of the third stage, the one that ResNet-50 has most of
        dict(conv("dense", 128, 14, 14, 256, 3, 256, input_relu=True), name="conv_14x14_256"),
        # the network's first layer: three channels, stride 2, a 7x7 window over raw pixels
        dict(conv("dense", 32, 224, 224, 3, 7, 64, stride=2, signed=True), name="stem_7x7_s2"),
        # a whole forward pass at a serving batch: 53 convolutions, shortcuts, pooling
        {"kind": "network", "net": "resnet50", "n": 8, "hw": 224, "table": "truncated", "name": "resnet50_b8"},
        # depthwise layer of the separable stack
        dict(conv("depthwise", 128, 56, 56, 144, 3, 1, table="noisy"), name="depthwise_56x56_144"),
        # a projection with channel counts that are multiples of nothing, on odd images
        dict(conv("dense", 37, 27, 31, 150, 1, 45, table="noisy", bias=True), name="pointwise_ragged"),
        # one training step of the layer-level caller: ranges and fake quantisation of the batch, forward, backward
        dict(conv("train", 32, 28, 28, 128, 3, 128), name="train_step_28x28_128"),
        # the first-generation op: uint8 codes in, int32 sums out
        dict(conv("quantised", 64, 28, 28, 64, 3, 96, table="noisy"), name="quantised_28x28_64"),
        # the reference's fp32 running total, for users who need its bits at a long K
        dict(conv("reference", 16, 14, 14, 256, 3, 256, table="noisy"), name="reference_order_14x14"),
    ]


MOST_MACS = {"dense": 2.5e10, "quantised": 1.2e10, "reference": 4e9, "train": 5e9, "depthwise": 6e8}


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["dense"] * 8 + ["depthwise"] * 2 + ["quantised", "reference", "train"])
    table = rng.choice(["truncated", "noisy", "exact"])
    h = _log(rng, 5, 112)
    w = max(4, h + rng.choice([0, 0, 0, -1, 1, 3]))
    if kind == "depthwise":
        c = rng.choice([_log(rng, 16, 400), 32 * rng.randint(1, 12), 4 * rng.randint(8, 96)])
        case = conv(kind, 1, h, w, c, rng.choice([3, 3, 3, 5]), 1, stride=rng.choice([1, 1, 2]), table=table, signed=rng.random() < 0.5)
    else:
        k = rng.choice([1, 1, 3, 3, 3, 5])
        c = rng.choice([_log(rng, 3, 512), 16 * rng.randint(1, 16), 64 * rng.randint(1, 8)])
        cout = rng.choice([_log(rng, 8, 512), 16 * rng.randint(1, 16), 64 * rng.randint(1, 8)])
        case = conv(kind, 1, h, w, c, k, cout, stride=rng.choice([1, 1, 1, 2]), table=table, signed=rng.random() < 0.5)
        if kind == "dense":
            case["padding"] = "VALID" if h > k and w > k and rng.random() < 0.2 else "SAME"
            case["dilation"] = 2 if k == 3 and min(h, w) > 8 and case["stride"] == 1 and rng.random() < 0.1 else 1
            case["input_relu"] = rng.random() < 0.4
            case["bias"] = rng.random() < 0.2
            case["residual"] = rng.random() < 0.2
            case["relu"] = rng.random() < 0.2
    per_image = macs(case)
    most = max(1, min(256, int(MOST_MACS[kind] / per_image), int(1.5e8 / (h * w * max(c, case["cout"])))))
    case["n"] = _log(rng, 1, most) if most > 1 else 1
    return case


def out_hw(case):
    def one(size):
        span = (case["k"] - 1) * case["dilation"] + 1
        return -(-size // case["stride"]) if case["padding"] == "SAME" else (size - span) // case["stride"] + 1
    return one(case["h"]), one(case["w"])


def macs(case):
    """Table lookups of one pass."""
    if case["kind"] == "network":
        return case["n"] * workloads.Network(case["net"], case["hw"]).macs_per_image()
    oh, ow = out_hw(case)
    return case["n"] * oh * ow * case["k"] ** 2 * case["c"] * case["cout"]


# ---------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------
def make_table(kind, seed):
    if kind == "noisy":
        return ax.noisy_table(seed)
    return ax.truncated_table() if kind == "truncated" else ax.exact_table()


def make_tensors(case, seed):
    """Activations (raw pixels: uniform; inside a network: a normal, seen through its ReLU unless that is left to the
    call), He-scaled filters and what is added to the output."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    n, h, w, c, k, cout = (case[x] for x in ("n", "h", "w", "c", "k", "cout"))
    if case["signed"]:
        x = torch.rand((n, h, w, c), generator=g, device=DEVICE) * 2 - 1
    else:
        x = torch.randn((n, h, w, c), generator=g, device=DEVICE)
        if not case["input_relu"]:
            x = x.clamp_(min=0)
    fan = k * k * (1 if case["kind"] == "depthwise" else c)
    f = torch.randn((k, k, c, cout), generator=g, device=DEVICE) * (2.0 / fan) ** 0.5
    oh, ow = out_hw(case)
    channels = c * cout if case["kind"] == "depthwise" else cout
    bias = torch.randn(channels, generator=g, device=DEVICE) if case["bias"] else None
    residual = torch.randn((n, oh, ow, channels), generator=g, device=DEVICE) if case["residual"] else None
    return x, f, bias, residual


def ranges_of(case, x, f):
    lo = 0.0 if case["input_relu"] or not case["signed"] else float(x.min())
    return lo, max(float(x.max()), 1e-3), float(f.min()), float(f.max())


def codes_of(case, seed):
    """uint8 operands of the quantised op and their ranges."""
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    x = (torch.randn((case["n"], case["h"], case["w"], case["c"]), generator=g, device=DEVICE) * 50 + 100).clamp_(0, 255).to(torch.uint8)
    f = (torch.randn((case["k"], case["k"], case["c"], case["cout"]), generator=g, device=DEVICE) * 35 + 128).clamp_(0, 255).to(torch.uint8)
    return x, f, (-1.0, 2.0, -0.5, 0.5)


def prepare(case, seed):
    if case["kind"] == "network":
        net = workloads.Network(case["net"], case["hw"])
        filters = workloads.make_filters(net.convs, seed)
        runner = workloads.GpuRunner(net, [make_table(case["table"], seed)], filters, DEVICE)
        g = torch.Generator(device=DEVICE).manual_seed(seed)
        x = torch.rand((case["n"], case["hw"], case["hw"], net.in_channels), generator=g, device=DEVICE) * 2 - 1
        runner.calibrate(x)
        return {"case": case, "runner": runner, "x": x}
    table = ax.Table(array=make_table(case["table"], seed))
    table.ensure_device(DEVICE.index)
    if case["kind"] == "quantised":
        x, f, r = codes_of(case, seed)
        return {"case": case, "table": table, "x": x, "f": f, "ranges": r}
    x, f, bias, residual = make_tensors(case, seed)
    if case["kind"] == "train":
        layer = ax.FakeApproxConv2D(case["c"], case["cout"], case["k"], strides=case["stride"], padding=case["padding"].lower(),
                                    mul_map_file=table).to(DEVICE).train()
        with torch.no_grad():
            layer.kernel.copy_(f)
        oh, ow = out_hw(case)
        g = torch.Generator(device=DEVICE).manual_seed(seed + 7)
        grad = torch.randn((case["n"], oh, ow, case["cout"]), generator=g, device=DEVICE)
        return {"case": case, "layer": layer, "x": x.requires_grad_(True), "grad": grad}
    return {"case": case, "table": table, "x": x, "f": f, "ranges": ranges_of(case, x, f), "bias": bias, "residual": residual}


# ---------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "network":
        return state["runner"].forward(state["x"])
    strides = [1, case["stride"], case["stride"], 1]
    if kind == "quantised":
        return ax.ax_conv2d(state["x"], state["f"], *state["ranges"], strides, case["padding"], table=state["table"], ax_tune=False)
    if kind == "train":
        layer, x = state["layer"], state["x"]
        x.grad = None
        layer.zero_grad(set_to_none=True)
        y = layer(x)
        y.backward(state["grad"])
        return {"y": y.detach(), "gx": x.grad, "gw": layer.kernel.grad, "gb": layer.bias.grad}
    if kind == "depthwise":
        return ax.approx_depthwise_conv2d_with_min_max_vars(state["x"], state["f"], *state["ranges"], strides, 8, state["table"],
                                                            case["padding"])
    return ax.approx_conv2d_with_min_max_vars(state["x"], state["f"], *state["ranges"], strides, 8, state["table"], case["padding"],
                                              dilations=(1, case["dilation"], case["dilation"], 1),
                                              accumulate="reference" if kind == "reference" else "exact", bias=state["bias"],
                                              residual=state["residual"], relu=case["relu"], input_relu=case["input_relu"])


def work(case):
    """Tensors in and out once; two operations per lookup.  A backward pass has twice the forward's."""
    if case["kind"] == "network":
        net = workloads.Network(case["net"], case["hw"])
        filters = 4 * sum(s.k * s.k * s.cin * s.cout for s, _ in net.convs)
        last, hw = net.convs[-1]
        return {"bytes": 4 * case["n"] * (case["hw"] ** 2 * net.in_channels + hw * hw * last.cout) + filters, "flops": 2 * macs(case)}
    oh, ow = out_hw(case)
    item = 1 if case["kind"] == "quantised" else 4
    channels = case["c"] * case["cout"] if case["kind"] == "depthwise" else case["cout"]
    n_in, n_f, n_out = case["n"] * case["h"] * case["w"] * case["c"], case["k"] ** 2 * case["c"] * case["cout"], case["n"] * oh * ow * channels
    if case["kind"] == "train":
        return {"bytes": 4 * (2 * n_in + 2 * n_f + 2 * n_out), "flops": 6 * macs(case)}
    return {"bytes": item * (n_in + n_f) + 4 * n_out * (2 if case["residual"] else 1), "flops": 2 * macs(case)}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantised":
        return "exact"              # whole numbers
    if kind == "reference":
        return "exact"              # the mode's purpose: every rounding of the reference's running total
    if kind == "train":
        return {"rel": 3e-3}        # the gradients are convolutions on the tensor cores in their default precision
    if kind == "network":
        return {"rel": 2e-3}        # a rounding in one layer may move a code in a later one
    # the sum of looked-up products is a whole number; what can differ are the fp32 sums of the taps and of the weights,
    # whose error grows with K (against 64 bits: 1.2e-6 at K = 64, 1.3e-5 at 576, 1e-4 at 4608) and which the
    # dequantisation partly cancels against the sum
    taps = case["k"] ** 2 * (1 if kind == "depthwise" else case["c"])
    return {"rel": 1e-6 + 1e-7 * taps}


# ---------------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------------
def _nudge(lo, hi):
    """{scale, 1/scale, offset} of a range in the op's fp32 arithmetic (it decides the codes)."""
    f = np.float32
    lo, hi = f(lo), f(hi)
    if lo == 0 and hi == 0:
        return f(0), f(0), f(0)
    s = (hi - lo) / f(255)
    z = f(0) - lo / s
    z = f(0) if z < 0 else f(255) if z > 255 else f(np.floor(np.abs(z) + f(0.5)) * np.sign(z))
    return s, f(1) / s, (f(0) - z) * s


def _codes(t, q):
    return ((t - float(q[2])) * float(q[1]) + 0.5).clamp(0, 255).to(torch.uint8)


def _window(case, size, out):
    span = (case["k"] - 1) * case["dilation"] + 1
    return max((out - 1) * case["stride"] + span - size, 0) // 2 if case["padding"] == "SAME" else 0


def _taps(case, x, fill):
    """(ky, kx, the tensor of taps [n, oh, ow, c]) for every window position."""
    oh, ow = out_hw(case)
    ph, pw = _window(case, case["h"], oh), _window(case, case["w"], ow)
    s, d, k = case["stride"], case["dilation"], case["k"]
    hh, ww = (oh - 1) * s + (k - 1) * d + 1, (ow - 1) * s + (k - 1) * d + 1
    p = torch.full((x.shape[0], max(hh, ph + case["h"]), max(ww, pw + case["w"]), x.shape[3]), fill, dtype=x.dtype, device=x.device)
    p[:, ph:ph + case["h"], pw:pw + case["w"]] = x
    for ky in range(k):
        for kx in range(k):
            yield ky, kx, p[:, ky * d:ky * d + (oh - 1) * s + 1:s, kx * d:kx * d + (ow - 1) * s + 1:s]


def _sums(case, lut, qx, qf, fill):
    """int64 [n*oh*ow, cout]: the sums of looked-up products."""
    oh, ow = out_hw(case)
    m = case["n"] * oh * ow
    lut = torch.from_numpy(lut.reshape(256, 256).astype(np.int64)).to(DEVICE)
    acc = torch.zeros((m, case["cout"]), dtype=torch.int64, device=DEVICE)
    for ky, kx, tap in _taps(case, qx, fill):
        rows = tap.reshape(m, case["c"]).t().contiguous().to(torch.int32)
        for c in range(case["c"]):
            acc += lut[:, qf[ky, kx, c].long()].index_select(0, rows[c])
    return acc


def exact(case, seed):
    kind = case["kind"]
    if kind == "network" or macs(case) > 3.2e10:
        return None                 # codes of later layers hang on the roundings of earlier ones
    lut = make_table(case["table"], seed)
    oh, ow = out_hw(case)
    m = case["n"] * oh * ow
    if kind == "quantised":
        x, f, r = codes_of(case, seed)
        zx, zf = int(-np.round(r[0] * 255.0 / (r[1] - r[0]))), int(-np.round(r[2] * 255.0 / (r[3] - r[2])))
        acc = _sums(case, lut, x, f, zx & 255)
        a = torch.zeros((m, 1), dtype=torch.int64, device=DEVICE)
        for _, _, tap in _taps(case, x, zx & 255):
            a += tap.reshape(m, case["c"]).sum(1, keepdim=True, dtype=torch.int64)
        b = f.sum((0, 1, 2), dtype=torch.int64)[None, :]
        kk = case["k"] ** 2 * case["c"]
        level = (r[1] - r[0]) / 255.0 * ((r[3] - r[2]) / 255.0)
        return (acc + kk * zx * zf - zf * a - zx * b).reshape(case["n"], oh, ow, -1), level * -2.0 ** 31, level * (2.0 ** 31 - 1)
    x, f, bias, residual = make_tensors(case, seed)
    if kind == "train":
        rng = (float(x.min()), float(x.max()), float(f.min()), float(f.max()))
        qx, qf = _nudge(*rng[:2]), _nudge(*rng[2:])
        seen = x
        x = _codes(x, qx).float() * float(qx[0]) + float(qx[2])
        f = _codes(f, qf).float() * float(qf[0]) + float(qf[2])
    else:
        x = x.clamp(min=0) if case["input_relu"] else x
        rng = ranges_of(case, x, f)
        qx, qf = _nudge(*rng[:2]), _nudge(*rng[2:])
    (s1, _, m1), (s2, _, m2) = [tuple(float(v) for v in q) for q in (qx, qf)]
    s1s2 = float(np.float32(s1) * np.float32(s2))
    zero = int(_codes(torch.zeros(1, device=DEVICE), qx))
    cx, cf = _codes(x, qx), _codes(f, qf)
    if kind == "depthwise":
        lut64 = torch.from_numpy(lut.reshape(256, 256).astype(np.int64)).to(DEVICE).reshape(-1)
        acc, a = 0, 0
        for (ky, kx, tap), (_, _, raw) in zip(_taps(case, cx, zero), _taps(case, x, 0.0)):
            a = a + raw.double()[..., None]
            acc = acc + lut64[(tap.long()[..., None] << 8) | cf[ky, kx].long()].double()
        kk = case["k"] ** 2
        b = f.double().sum((0, 1))
        y = s1s2 * acc + m2 * a + m1 * b - kk * m1 * m2
        return y.reshape(case["n"], oh, ow, -1)
    acc = _sums(case, lut, cx, cf, zero).double()
    a = torch.zeros((m, 1), dtype=torch.float64, device=DEVICE)
    for _, _, tap in _taps(case, x, 0.0):
        a += tap.reshape(m, case["c"]).sum(1, keepdim=True, dtype=torch.float64)
    kk = case["k"] ** 2 * case["c"]
    y = (s1s2 * acc + m2 * a + m1 * f.double().sum((0, 1, 2))[None, :] - kk * m1 * m2).reshape(case["n"], oh, ow, -1)
    if kind == "train":
        g = torch.Generator(device=DEVICE).manual_seed(seed + 7)
        grad = torch.randn((case["n"], oh, ow, case["cout"]), generator=g, device=DEVICE).double()
        gx, gw = torch.zeros_like(seen, dtype=torch.float64), torch.zeros_like(f, dtype=torch.float64)
        ph, pw = _window(case, case["h"], oh), _window(case, case["w"], ow)
        s, k = case["stride"], case["k"]
        pad = torch.zeros((case["n"], max((oh - 1) * s + k, ph + case["h"]), max((ow - 1) * s + k, pw + case["w"]), case["c"]),
                          dtype=torch.float64, device=DEVICE)
        for ky, kx, tap in _taps(case, x.double(), 0.0):
            gw[ky, kx] = tap.reshape(m, -1).t() @ grad.reshape(m, -1)
            pad[:, ky:ky + (oh - 1) * s + 1:s, kx:kx + (ow - 1) * s + 1:s] += grad @ f[ky, kx].double().t()
        gx = pad[:, ph:ph + case["h"], pw:pw + case["w"]].contiguous()
        return {"y": y, "gx": gx, "gw": gw, "gb": grad.sum((0, 1, 2))}
    if bias is not None:
        y = y + bias.double()
    if residual is not None:
        y = y + residual.double()
    return y.clamp(min=0) if case["relu"] else y
