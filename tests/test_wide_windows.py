"""Wide windows with wide dilations, of which one output pixel's taps nearly fill the shared memory that the expanded tables'
preparation has: they are served by the expanded tables up to the last channel count whose taps fit."""
import numpy as np
import pytest

# k, dilation, channel counts whose taps fit the 220 KiB without their codes only (and are no multiple of 4: those have their pieces
# apart), and one that does not fit at all
FAMILIES = [(3, 18, range(33, 40), 64), (3, 12, (81, 82, 83), 121), (11, 2, (113,), 160), (5, 12, range(19, 23), 40), (11, 8, (7,), 12), (2, 30, range(49, 56), 80)]


@pytest.mark.parametrize("k,dil,fit,too_many", FAMILIES, ids=str)
def test_windows_whose_taps_fit_have_scratch(built, k, dil, fit, too_many):
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import ops
    t = ax.Table(array=ax.noisy_table(3))

    def scratch(c):
        return ops.fast_workspace_bytes((4, 64, 64, c), (k, k, c, 64), [1, 1, 1, 1], "SAME", (1, dil, dil, 1), t)
    assert all(scratch(c) > 0 for c in fit if c % 4) and scratch(too_many) == 0


# n, h, w, c, k, cout, dilation, padding: no room for the codes; the last two beside a family's first, where there is
SHAPES = [(1, 40, 41, 33, 3, 24, 18, "SAME"), (4, 60, 61, 39, 3, 24, 18, "VALID"), (2, 33, 30, 83, 3, 16, 12, "SAME"), (1, 24, 25, 113, 11, 8, 2, "SAME"),
          (2, 64, 60, 20, 5, 8, 12, "SAME"), (2, 112, 112, 7, 11, 16, 8, "VALID"), (1, 40, 41, 32, 3, 24, 18, "SAME"), (1, 24, 25, 112, 11, 8, 2, "SAME")]


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["noisy", "truncated", "exact"])
@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_they_match_the_checker(built, shape, kind):
    import torch
    import tf_approximate_b200 as ax
    from oracle import oracle as O
    n, h, w, c, k, co, dil, pad = shape
    lut = {"truncated": ax.truncated_table(), "noisy": ax.noisy_table(4), "exact": ax.exact_table()}[kind]
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape[:6])))
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.7, 1.0, float(f.min()), float(f.max()))
    d = O.desc(n, h, w, c, k, k, co, (1, 1), (dil, dil), pad)
    ref = O.conv2d(d, lut, x, f, *mm, want=("out_exact", "acc"))
    y, dbg = ax.approx_conv2d_with_min_max_vars(torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), *mm, [1, 1, 1, 1], 8, t, pad,
                                                dilations=[1, dil, dil, 1], debug=True)
    assert dbg["plan"]["route"]["kernels"] == "expanded" and dbg["plan"]["status"] == 0
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_exact"].view(np.uint32))
