"""GPU: the reference's order of additions on expanded tables (accumulate="reference" without a caller's buffer), bit for bit
against the CPU checker's fp32 running total and against the kernel that a plan-sized buffer selects: one to four pixels per
lane, ragged tiles of pixels and channels, im2col rows, dilation, sums far beyond 2^24."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# n, h, w, c, k, cout, stride, dilation, padding
SHAPES = [
    (1, 9, 9, 512, 3, 200, 1, 1, "SAME"),
    (1, 1, 33, 2048, 1, 128, 1, 1, "SAME"),
    (4, 40, 40, 3, 11, 40, 1, 1, "SAME"),
    (2, 23, 29, 150, 3, 45, 2, 2, "VALID"),
    (3, 100, 101, 32, 3, 13, 1, 1, "SAME"),
    (16, 14, 14, 64, 3, 264, 1, 1, "SAME"),
    (9, 130, 129, 20, 5, 8, 1, 1, "SAME"),
]


@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_reference_order_on_expanded_tables(built, shape):
    import torch
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import _lib, ops
    n, h, w, c, k, co, s, dil, pad = shape
    lut = ax.noisy_table(9)
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape[:6])))
    x = rng.uniform(0, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.1, 1.0, float(f.min()) / 2, float(f.max()))
    size, desc = C.c_size_t(), _lib.ConvDesc(n, h, w, c, k, k, c, co, s, s, dil, dil, 0 if pad == "SAME" else 1, 0, 1, 1)
    assert _lib.load().axc_conv2d_fast_workspace_bytes(t.handle, C.byref(desc), C.byref(size)) == 0 and size.value > 0
    ref = O.conv2d(O.desc(n, h, w, c, k, k, co, (s, s), (dil, dil), pad), lut, x, f, *mm, want=("out_ref", "out_exact"))
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    args = (*mm, [1, s, s, 1], 8, t, pad)
    opts = {"dilations": [1, dil, dil, 1], "accumulate": "reference"}
    y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *args, debug=True, **opts)
    assert dbg["plan"]["status"] == 0
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_ref"].view(np.uint32))
    assert not np.array_equal(ref["out_ref"], ref["out_exact"]) or k * k * c < 2000
    ws = torch.zeros(ops.workspace_bytes(x.shape, f.shape, [1, s, s, 1], pad, (1, dil, dil, 1)), dtype=torch.uint8, device="cuda")
    y2, dbg2 = ax.approx_conv2d_with_min_max_vars(xd, fd, *args, debug=True, workspace=ws, **opts)
    assert torch.equal(y.view(torch.int32), y2.view(torch.int32)) and torch.equal(dbg["acc"], dbg2["acc"])
    assert torch.equal(dbg["qfilter"], dbg2["qfilter"]) and torch.equal(dbg["qinput"], dbg2["qinput"])
    g = torch.Generator(device="cuda").manual_seed(1)
    bias, res = torch.randn(co, device="cuda", generator=g), torch.randn(y.shape, device="cuda", generator=g)
    z = ax.approx_conv2d_with_min_max_vars(xd, fd, *args, bias=bias, residual=res, relu=True, **opts)
    assert torch.equal(z.view(torch.int32), torch.relu(y + bias + res).view(torch.int32))
