"""GPU: sums of columns of matrices that are much wider than they are long, narrower than a warp, or a single column, against 64
bits; and their launches: up to 256 rows need one kernel however wide the matrix is."""
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 100000), (64, 30000), (256, 4100), (257, 4100), (49, 2048), (3211264, 1), (200704, 3), (1048576, 16), (1025, 1), (1024, 2), (5000, 31), (5000, 32), (5000, 34), (70001, 128), (300, 124)]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("rows,cols", SHAPES)
def test_column_sums(built, rows, cols, offset):
    import torch
    from tf_approximate_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows * cols + offset, device="cuda", generator=g)[offset:].view(rows, cols)     # also 4 bytes past a 16-byte boundary
    before = ops.launch_count()
    got = ops.column_sums(x)
    launches = ops.launch_count() - before
    # a tree of chains of at most rows / 2368 + 60 additions of fp32: each loses half a unit of what is added so far
    bound = x.double().abs().sum(0) * (rows / 2368 + 60) * 2.0 ** -24
    assert bool(((got.double() - x.double().sum(0)).abs() <= bound).all())
    assert launches == 1 if rows <= 256 else launches <= 2
