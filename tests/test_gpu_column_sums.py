"""GPU: sums of columns (the gradient of a bias) against 64 bits, at the edges of the kernel's blocks, warps and column tiles."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("rows,cols", [(0, 5), (1, 1), (7, 128), (8, 129), (9, 4), (2367, 33), (2369, 132), (25088, 128), (100003, 3), (12, 2000)])
def test_column_sums(built, rows, cols, offset):
    import torch
    from tf_approximate_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    x = torch.randn(rows * cols + offset, device="cuda", generator=g)[offset:].view(rows, cols)     # also 4 bytes past a 16-byte boundary
    got = ops.column_sums(x)
    assert got.shape == (cols,)
    # every sum is a tree of chains of at most rows / 2368 + 60 additions of fp32: each loses half a unit of what is added so far
    bound = x.double().abs().sum(0) * (rows / 2368 + 60) * 2.0 ** -24
    assert bool(((got.double() - x.double().sum(0)).abs() <= bound).all())
