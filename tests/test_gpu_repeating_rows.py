"""GPU: one-byte expanded tables whose rows repeat every 64 activations (truncated products) and ones whose rows do not, against the
CPU checker, bit for bit: every tile, tables from global memory and made by the CTAs, one chunk of K and several more than the ring of
tables holds, K split over CTAs, several units per CTA."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# n, h, w, c, k, cout
SHAPES = [
    (1, 7, 7, 512, 3, 512), (1, 64, 64, 16, 1, 160), (2, 20, 20, 32, 3, 64), (1, 30, 30, 512, 1, 24), (4, 56, 57, 32, 3, 64), (8, 28, 28, 64, 1, 256),
    (3, 61, 67, 48, 3, 40), (20, 97, 97, 32, 3, 8), (12, 149, 149, 16, 1, 24), (12, 149, 149, 20, 1, 24), (1, 64, 64, 3, 7, 64), (9, 14, 14, 256, 1, 500),
]


def tables(ax):
    rng = np.random.Generator(np.random.PCG64(12))
    noise = rng.integers(0, 251, 65536)
    exact = ax.exact_table().astype(np.int64)
    late = ax.truncated_table().astype(np.int64)
    late[255 * 256 + 9] += 1                        # one entry short of repeating
    return {"cleared 6": ax.truncated_table(), "cleared 2": ax.truncated_table(2), "any": np.clip(exact + noise - 100, 0, 65535).astype(np.uint16),
            "late": late.astype(np.uint16)}


@pytest.mark.parametrize("kind", ["cleared 6", "cleared 2", "any", "late"])
@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_rows_that_repeat(built, shape, kind):
    import torch
    import tf_approximate_b200 as ax
    n, h, w, c, k, co = shape
    lut = tables(ax)[kind]
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape)))
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.7, 1.0, float(f.min()), float(f.max()))
    ref = O.conv2d(O.desc(n, h, w, c, k, k, co), lut, x, f, *mm, want=("out_exact", "acc"))
    xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
    y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, 1, 1, 1], 8, t, "SAME", debug=True)
    assert dbg["plan"]["route"]["kernels"] == "expanded" and dbg["plan"]["status"] == 0
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_exact"].view(np.uint32))
    z = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, 1, 1, 1], 8, t, "SAME")      # (the plain end of a tile)
    assert torch.equal(z.view(torch.int32), y.view(torch.int32))
