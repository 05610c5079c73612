"""GPU: the expanded-table depthwise kernel's shares of columns - less than a column per warp, pieces of one column, shares that
end inside a band - against the CPU checker, bit for bit, by TMA and by plain loads."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# n, h, w, c, stride: the smallest calls that the kernel takes, narrow images, several bands per warp, no TMA (33 channels)
SHAPES = [(1, 32, 32, 32, 1), (1, 8, 128, 32, 1), (64, 9, 5, 36, 1), (300, 3, 4, 40, 1), (4, 57, 55, 144, 1), (1, 64, 64, 32, 2), (70, 9, 11, 36, 2),
          (2, 61, 59, 96, 2), (2, 40, 41, 33, 1), (3, 45, 47, 33, 2)]


@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_shares_of_columns(built, shape):
    import torch
    import tf_approximate_b200 as ax
    n, h, w, c, s = shape
    lut = ax.noisy_table(6)
    rng = np.random.Generator(np.random.PCG64(sum(shape)))
    x = rng.uniform(-1, 2, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.3, (3, 3, c, 1)).astype(np.float32)
    mm = (-1.0, 2.0, float(f.min()), float(f.max()))
    ref = O.depthwise_conv2d(O.desc(n, h, w, c, 3, 3, 1, (s, s)), lut, x, f, *mm)
    xd, fd, t = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), ax.Table(array=lut)
    y, dbg = ax.approx_depthwise_conv2d_with_min_max_vars(xd, fd, *mm, [1, s, s, 1], 8, t, "SAME", debug=True)
    z = ax.approx_depthwise_conv2d_with_min_max_vars(xd, fd, *mm, [1, s, s, 1], 8, t, "SAME")
    assert dbg["status"] == 0
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_ref"].view(np.uint32)) and torch.equal(y, z)
