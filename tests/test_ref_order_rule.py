"""Which reference-order calls take the expanded tables: not those with so many channel tiles for their few pixels that the GPU has to
go round more often than on the kernel that looks entries up one by one."""
import ctypes as C

import numpy as np
import pytest

NONE, PLAN, COMMON_K, EXPANDED = range(4)

# n, h, w, c, k, cout; and the neighbours with one round only
SLOWER = [(1, 1, 1, 2048, 1, 4096), (1, 7, 7, 512, 1, 2048), (4, 7, 7, 512, 1, 2048), (1, 5, 5, 64, 3, 2400)]
FASTER = [(1, 1, 1, 16384, 1, 1024), (1, 7, 7, 512, 1, 1184), (16, 7, 7, 512, 1, 2048), (1, 5, 5, 512, 3, 128)]


def ask(table, shape, plan, nbytes=None):
    from tf_approximate_b200 import _lib
    L = _lib.load()
    n, h, w, c, k, cout = shape
    d = _lib.ConvDesc(n, h, w, c, k, k, c, cout, 1, 1, 1, 1, 0, 0, 1, plan)
    if nbytes is not None:
        out = (C.c_int32 * 4)()
        assert L.axc_conv2d_route(table.handle, C.byref(d), nbytes, out) == 0
        return out[0]
    general, fast, any_table = C.c_size_t(), C.c_size_t(), C.c_size_t()
    assert L.axc_conv2d_workspace_bytes(C.byref(d), C.byref(general)) == 0
    assert L.axc_conv2d_fast_workspace_bytes(table.handle, C.byref(d), C.byref(fast)) == 0
    assert L.axc_conv2d_fast_workspace_bytes(None, C.byref(d), C.byref(any_table)) == 0
    return general.value, fast.value, any_table.value


def test_the_rule_and_its_sizes(built):
    import tf_approximate_b200 as ax
    t = ax.Table(array=ax.noisy_table(3))
    for shape in SLOWER:
        for plan in (0, 1):
            general, fast, any_table = ask(t, shape, plan)
            assert fast == 0 and any_table > 0, shape
            assert ask(t, shape, plan, general) == COMMON_K and ask(t, shape, plan, general + any_table) == COMMON_K
            # a buffer of the size that serves every table is not refused
            if any_table < general:
                assert ask(t, shape, plan, any_table) == EXPANDED
    assert any(ask(t, s, 1)[2] < ask(t, s, 1)[0] for s in SLOWER)
    for shape in FASTER:
        fast = ask(t, shape, 1)[1]
        assert fast > 0 and ask(t, shape, 1, fast) == EXPANDED, shape


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SLOWER + FASTER[1:], ids=["-".join(str(v) for v in s) for s in SLOWER + FASTER[1:]])
def test_both_sides_match_the_checker(built, shape):
    import torch
    import tf_approximate_b200 as ax
    from oracle import oracle as O
    n, h, w, c, k, co = shape
    lut = ax.noisy_table(9)
    t = ax.Table(array=lut)
    rng = np.random.Generator(np.random.PCG64(sum(shape)))
    x = rng.uniform(0, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
    mm = (-0.1, 1.0, float(f.min()) / 2, float(f.max()))
    want = O.conv2d(O.desc(n, h, w, c, k, k, co, (1, 1), (1, 1), "SAME"), lut, x, f, *mm, want=("out_ref",))["out_ref"]
    for plan in ("keep", "none"):
        y, dbg = ax.approx_conv2d_with_min_max_vars(torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), *mm, [1, 1, 1, 1], 8, t, "SAME",
                                                    accumulate="reference", plan=plan, debug=True)
        assert dbg["plan"]["route"]["kernels"] == ("common-k" if shape in SLOWER else "expanded")
        assert shape in SLOWER or dbg["plan"]["status"] == 0          # (the other kernel has no header)
        assert np.array_equal(y.cpu().numpy().view(np.uint32), want.view(np.uint32))
