"""GPU: the preparation of the expanded-table kernels (codes, patch sums, filter sums, weight lists) against the CPU checker, bit for
bit, where its tiles and loops can go wrong: rows wider than a tile, im2col rows with dilation and a single channel, channel
counts that are no multiple of 4 or 16, long chains of additions, several tiles per image."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# n, h, w, c, k, cout, stride, dilation, padding
SHAPES = [
    (1, 3, 1400, 8, 1, 256, 1, 1, "SAME"),
    (2, 33, 40, 3, 5, 64, 1, 3, "SAME"),
    (1, 64, 64, 1, 9, 40, 1, 1, "VALID"),
    (2, 20, 20, 36, 3, 40, 1, 1, "SAME"),
    (3, 31, 29, 66, 3, 32, 2, 1, "SAME"),
    (1, 7, 7, 500, 3, 50, 1, 1, "SAME"),
    (1, 14, 14, 2048, 1, 64, 1, 1, "SAME"),
    (5, 27, 25, 21, 3, 33, 1, 1, "VALID"),
    (2, 56, 56, 64, 3, 48, 2, 2, "SAME"),
]


@pytest.mark.parametrize("kind", ["truncated", "noisy", "exact"])
@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_preparation_matches_the_checker(built, shape, kind):
    import torch
    import tf_approximate_b200 as ax
    n, h, w, c, k, co, s, dil, pad = shape
    lut = {"truncated": ax.truncated_table(), "noisy": ax.noisy_table(4), "exact": ax.exact_table()}[kind]
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape[:6])))
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.7, 1.0, float(f.min()), float(f.max()))
    d = O.desc(n, h, w, c, k, k, co, (s, s), (dil, dil), pad)
    for relu in (False, True):
        seen = np.maximum(x, 0) if relu else x
        ref = O.conv2d(d, lut, seen, f, *mm, want=("out_exact", "acc"))
        y, dbg = ax.approx_conv2d_with_min_max_vars(torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), *mm, [1, s, s, 1], 8, t, pad,
                                                    dilations=[1, dil, dil, 1], input_relu=relu, debug=True)
        assert dbg["plan"]["route"]["kernels"] == "expanded" and dbg["plan"]["status"] == 0
        assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
        assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_exact"].view(np.uint32))
    if dil == 1:
        a, b = rng.integers(0, 256, x.shape).astype(np.uint8), rng.integers(0, 256, f.shape).astype(np.uint8)
        q, _, _ = ax.ax_conv2d(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), -1.0, 2.0, -0.5, 0.5, [1, s, s, 1], pad, table=t, ax_tune=False)
        assert np.array_equal(q.cpu().numpy(), O.qconv2d(d, lut, a, b, O.quantized_zero_point(-1.0, 2.0), O.quantized_zero_point(-0.5, 0.5)))
