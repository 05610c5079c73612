"""GPU: the expanded-table kernels against the CPU checker, bit for bit, at the sizes where they can go wrong: channel tiles
(8 / 16), K chunks (16), codes in pixel order and as im2col rows, K split over CTAs, tables built by the CTAs and taken from global
memory, and every form a table can be kept in, with small pixel tiles (SHAPES); edges of the larger ones and CTAs that go from
unit to unit (TILES)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def tables(ax):
    rng = np.random.Generator(np.random.PCG64(8))
    return {"exact": ax.exact_table(), "offset": (ax.exact_table() + 7).astype(np.uint16), "byte": ax.truncated_table(), "digits": rng.integers(0, 65280, 65536).astype(np.uint16),
            "centred": ax.noisy_table(3), "neither": rng.integers(0, 65536, 65536).astype(np.uint16)}


# n, h, w, c, kh, kw, cout, stride, dilation, padding
SHAPES = [
    (1, 7, 7, 512, 3, 3, 512, 1, 1, "SAME"),        # 49 pixels, K split over CTAs
    (2, 32, 32, 16, 3, 3, 32, 1, 1, "SAME"),        # whole 16-byte pieces
    (3, 27, 31, 150, 1, 1, 45, 1, 1, "SAME"),       # ragged channels on both sides
    (1, 64, 64, 3, 7, 7, 64, 2, 1, "SAME"),         # im2col rows
    (1, 112, 112, 8, 3, 3, 32, 1, 1, "SAME"),       # im2col rows, 16-byte input pixels
    (2, 40, 37, 32, 3, 3, 24, 1, 2, "SAME"),        # dilation
    (7, 33, 29, 20, 3, 3, 33, 2, 1, "VALID"),       # stride without padding
    (1, 14, 14, 1024, 1, 1, 256, 2, 1, "SAME"),     # input pixels that no window reads
    (4, 56, 57, 32, 3, 3, 64, 1, 1, "SAME"),        # enough pixels for tables in global memory
    (9, 37, 37, 64, 1, 1, 72, 1, 1, "SAME"),
]


@pytest.mark.parametrize("kind", ["exact", "offset", "byte", "digits", "centred", "neither"])
@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_expanded_tables_match_the_checker(built, shape, kind):
    import torch
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import ops
    n, h, w, c, kh, kw, co, s, d, pad = shape
    lut = tables(ax)[kind]
    t = ax.Table(array=lut)
    fast = ops.fast_workspace_bytes((n, h, w, c), (kh, kw, c, co), [1, s, s, 1], pad, (1, d, d, 1), t)
    assert (fast > 0) == (kind != "neither")
    rng = np.random.Generator(np.random.PCG64(sum(shape[:8])))
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (kh, kw, c, co)).astype(np.float32)
    mm = (-0.7, 1.0, float(f.min()), float(f.max()))
    ref = O.conv2d(O.desc(n, h, w, c, kh, kw, co, (s, s), (d, d), pad), lut, x, f, *mm, want=("out_exact", "acc"))
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    call = lambda *a, **kw_: ax.approx_conv2d_with_min_max_vars(xd, fd, *a, [1, s, s, 1], 8, t, pad, dilations=(1, d, d, 1), **kw_)  # noqa: E731
    y, dbg = call(*mm, debug=True)
    assert dbg["plan"]["status"] == 0
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    want = torch.from_numpy(ref["out_exact"]).cuda()
    assert torch.equal(y.view(torch.int32), want.view(torch.int32))
    # the plain call (another end of the kernel), ranges on the device, and what rides along with a call
    assert torch.equal(call(*mm).view(torch.int32), want.view(torch.int32))
    assert torch.equal(call(*[torch.tensor(v, device="cuda") for v in mm]).view(torch.int32), want.view(torch.int32))
    g = torch.Generator(device="cuda").manual_seed(1)
    bias, res = torch.randn(co, device="cuda", generator=g), torch.randn(want.shape, device="cuda", generator=g)
    fused = call(*mm, bias=bias, residual=res, relu=True)
    assert torch.equal(fused.view(torch.int32), torch.relu(want + bias + res).view(torch.int32))
    # the plan-based kernels, which a workspace of their size selects
    ws = torch.zeros(ops.workspace_bytes((n, h, w, c), (kh, kw, c, co), [1, s, s, 1], pad, (1, d, d, 1)), dtype=torch.uint8, device="cuda")
    (a, da), (b, db) = call(*mm, input_relu=True, debug=True), call(*mm, input_relu=True, workspace=ws, debug=True)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))
    assert da["plan"]["route"]["kernels"] == ("plan" if kind == "neither" else "expanded") and db["plan"]["route"]["kernels"] == "plan"


# n, h, w, c, k, cout, form, pixels per tile, tables from global memory, K split; at least as many units as fill 148 CTAs more
# than once, and a ragged last tile and channel tile
TILES = [
    (40, 97, 97, 20, 1, 8, "byte", 1024, True, False),
    (12, 149, 149, 20, 1, 24, "byte", 2048, True, False),
    (20, 97, 97, 32, 3, 8, "byte", 2048, True, True),
    (40, 97, 97, 16, 1, 8, "byte", 1024, False, False),
    (12, 149, 149, 16, 1, 24, "byte", 2048, False, False),
    (12, 149, 149, 16, 1, 24, "exact", 2048, False, False),
    (40, 97, 97, 64, 1, 13, "digits", 1024, True, False),
    (12, 149, 149, 20, 1, 13, "digits", 2048, True, False),
    (12, 149, 149, 20, 1, 13, "centred", 2048, True, False),
    (12, 149, 149, 16, 1, 13, "digits", 2048, False, False),
    (40, 97, 97, 16, 1, 13, "digits", 3072, True, False),
    (40, 97, 97, 16, 1, 13, "centred", 3072, True, False),
]


@pytest.mark.parametrize("shape", TILES, ids=["-".join(str(v) for v in s) for s in TILES])
def test_large_tiles_and_several_units_per_cta(built, shape):
    import torch
    import tf_approximate_b200 as ax
    n, h, w, c, k, co, kind, tile, in_global, split = shape
    lut = tables(ax)[kind]
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape[:6])))
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.7, 1.0, float(f.min()), float(f.max()))
    d = O.desc(n, h, w, c, k, k, co)
    ref = O.conv2d(d, lut, x, f, *mm, want=("out_exact", "acc"))
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, 1, 1, 1], 8, t, "SAME", debug=True)
    route = dbg["plan"]["route"]
    assert dbg["plan"]["status"] == 0
    assert (route["kernels"], route["tile"], route["tables_in_global_memory"], route["splits"] > 1) == ("expanded", tile, in_global, split)
    units = -(-n * h * w // tile) * -(-co // (16 if kind in ("byte", "exact") else 8)) * route["splits"]
    assert units > 148 and n * h * w % tile
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    want = torch.from_numpy(ref["out_exact"]).cuda()
    assert torch.equal(y.view(torch.int32), want.view(torch.int32))
    res = torch.flip(want, [0])
    fused = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, 1, 1, 1], 8, t, "SAME", residual=res, relu=True)
    assert torch.equal(fused.view(torch.int32), torch.relu(want + res).view(torch.int32))
    a, b = rng.integers(0, 256, x.shape).astype(np.uint8), rng.integers(0, 256, f.shape).astype(np.uint8)
    q, _, _ = ax.ax_conv2d(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), -1.0, 2.0, -0.5, 0.5, [1, 1, 1, 1], "SAME", table=t, ax_tune=False)
    assert np.array_equal(q.cpu().numpy(), O.qconv2d(d, lut, a, b, O.quantized_zero_point(-1.0, 2.0), O.quantized_zero_point(-0.5, 0.5)))


def test_a_table_without_a_form_keeps_its_plan(built):
    """A table that fits none of the forms is served by the plan-based kernels, whose plan survives from call to call."""
    import torch
    import tf_approximate_b200 as ax
    g = torch.Generator(device="cuda").manual_seed(4)
    x = torch.rand((2, 40, 40, 32), device="cuda", generator=g)
    f = torch.randn((3, 3, 32, 48), device="cuda", generator=g)
    t = ax.Table(array=tables(ax)["neither"])
    rebuilt = [ax.approx_conv2d_with_min_max_vars(x, f, 0.0, 1.0, -3.0, 3.0, [1, 1, 1, 1], 8, t, "SAME", debug=True)[1]["plan"]["rebuilt"]
               for _ in range(3)]
    assert rebuilt == [1, 0, 0]


def test_unusual_values_and_addresses(built):
    """NaN, infinities and values outside the range; an input that starts 4 bytes past a 16-byte boundary; a one-value range."""
    import torch
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(2)
    x = torch.rand((2, 40, 40, 32), device="cuda", generator=g) * 2 - 1
    x.view(-1)[::997] = float("nan"); x.view(-1)[1::991] = float("inf"); x.view(-1)[2::983] = -float("inf"); x.view(-1)[3::977] = 7.0
    f = torch.randn((3, 3, 32, 48), device="cuda", generator=g) * 0.1
    t = ax.Table(array=ax.noisy_table(5))
    odd = torch.empty(x.numel() + 1, device="cuda")[1:].view(x.shape).copy_(x)
    for mm in [(-1.0, 1.0, -0.3, 0.3), (0.0, 0.0, -0.3, 0.3), (0.25, 0.75, 0.0, 0.0)]:
        ws = torch.zeros(ops.workspace_bytes(x.shape, f.shape, [1, 1, 1, 1], "SAME"), dtype=torch.uint8, device="cuda")
        want = ax.approx_conv2d_with_min_max_vars(x, f, *mm, [1, 1, 1, 1], 8, t, "SAME", workspace=ws)
        for inp in (x, odd):
            y = ax.approx_conv2d_with_min_max_vars(inp, f, *mm, [1, 1, 1, 1], 8, t, "SAME")
            assert torch.equal(torch.isnan(y), torch.isnan(want))
            assert torch.equal(torch.nan_to_num(y, 0.0).view(torch.int32), torch.nan_to_num(want, 0.0).view(torch.int32))


Q_SHAPES = [  # n, h, w, c, k, cout, stride, padding, input range, filter range
    (2, 28, 28, 64, 3, 96, 1, "SAME", (-1.0, 2.0), (-0.5, 0.5)),
    (9, 21, 23, 30, 3, 45, 2, "SAME", (0.5, 2.0), (-0.5, 0.25)),        # zero point of the input below 0: padded taps wrap
    (2, 50, 50, 3, 5, 50, 1, "VALID", (0.0, 1.0), (0.0, 1.0)),          # im2col rows, no zero-point terms
    (5, 50, 51, 32, 3, 64, 1, "SAME", (-3.0, -1.0), (-1.0, 3.0)),
]


@pytest.mark.parametrize("kind", ["exact", "offset", "byte", "digits", "centred"])
@pytest.mark.parametrize("shape", Q_SHAPES, ids=["-".join(str(v) for v in s[:8]) for s in Q_SHAPES])
def test_quantised_operands(built, shape, kind):
    """uint8 operands on the expanded tables, the zero-point terms added at the end, against the checker's functor."""
    import ctypes as C
    import torch
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import _lib
    n, h, w, c, k, co, s, pad, ri, rf = shape
    lut = tables(ax)[kind]
    rng = np.random.Generator(np.random.PCG64(77 + c))
    a = rng.integers(0, 256, (n, h, w, c)).astype(np.uint8)
    b = rng.integers(0, 256, (k, k, c, co)).astype(np.uint8)
    zi, zf = O.quantized_zero_point(*ri), O.quantized_zero_point(*rf)
    t = ax.Table(array=lut)
    size, out = C.c_size_t(), (C.c_int32 * 4)()
    desc = _lib.ConvDesc(n, h, w, c, k, k, c, co, s, s, 1, 1, 0 if pad == "SAME" else 1, 0, 0, 1)
    assert _lib.load().axc_qconv2d_fast_workspace_bytes(t.handle, C.byref(desc), C.byref(size)) == 0 and size.value > 0
    assert _lib.load().axc_qconv2d_route(t.handle, C.byref(desc), size.value, out) == 0 and out[0] == 3
    ref = O.qconv2d(O.desc(n, h, w, c, k, k, co, (s, s), (1, 1), pad), lut, a, b, zi, zf)
    y, _, _ = ax.ax_conv2d(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), *ri, *rf, [1, s, s, 1], pad, table=t,
                           ax_tune=False)
    assert np.array_equal(y.cpu().numpy(), ref)
