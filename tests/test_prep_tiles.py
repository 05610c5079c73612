"""GPU: the preparation's tiles that are 7 and 8 pixels wide, or that fill a warp's lanes with a part of a row, against the CPU checker bit for
bit: codes, sums and outputs of the layers that have them."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# n, h, w, c, k, cout, stride, padding
SHAPES = [(5, 28, 28, 512, 1, 16, 1, "SAME"), (2, 56, 56, 256, 1, 16, 1, "SAME"), (3, 14, 15, 1024, 1, 24, 1, "SAME"), (2, 45, 45, 37, 5, 20, 1, "SAME"),
          (2, 61, 60, 100, 3, 17, 1, "VALID"), (1, 75, 74, 80, 3, 33, 2, "SAME"), (40, 13, 13, 12, 3, 16, 1, "SAME"), (1, 500, 9, 24, 3, 16, 1, "SAME"), (4, 19, 700, 20, 1, 48, 2, "SAME")]


@pytest.mark.parametrize("kind", ["noisy", "exact"])
@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_tiles_match_the_checker(built, shape, kind):
    import torch
    import tf_approximate_b200 as ax
    n, h, w, c, k, co, s, pad = shape
    lut = {"noisy": ax.noisy_table(4), "exact": ax.exact_table()}[kind]
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape[:6])))
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.7, 1.0, float(f.min()), float(f.max()))
    d = O.desc(n, h, w, c, k, k, co, (s, s), (1, 1), pad)
    ref = O.conv2d(d, lut, x, f, *mm, want=("out_exact", "acc"))
    y, dbg = ax.approx_conv2d_with_min_max_vars(torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), *mm, [1, s, s, 1], 8, t, pad, debug=True)
    assert dbg["plan"]["route"]["kernels"] == "expanded" and dbg["plan"]["status"] == 0
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_exact"].view(np.uint32))
    a, b = rng.integers(0, 256, x.shape).astype(np.uint8), rng.integers(0, 256, f.shape).astype(np.uint8)
    q, _, _ = ax.ax_conv2d(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), -1.0, 2.0, -0.5, 0.5, [1, s, s, 1], pad, table=t, ax_tune=False)
    assert np.array_equal(q.cpu().numpy(), O.qconv2d(d, lut, a, b, O.quantized_zero_point(-1.0, 2.0), O.quantized_zero_point(-0.5, 0.5)))
