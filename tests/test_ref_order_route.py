"""The route of a call whose sum is taken in the reference's order: where the expanded tables serve it the route says so, with the
tile of that kernel, and the status that it leaves behind a kept plan is the one that debug=True reads."""
import ctypes as C

import pytest

NONE, PLAN, COMMON_K, EXPANDED = range(4)

# n, h, w, c, k, cout: a scratch larger than the plan and one that is not
SHAPES = [(16, 14, 14, 256, 3, 256), (1, 14, 14, 1024, 1, 512), (9, 130, 129, 20, 5, 8)]


def ask(table, shape, plan, nbytes=None, accumulate=1):
    """{general bytes, fast bytes}, or with `nbytes` the route."""
    from tf_approximate_b200 import _lib
    L = _lib.load()
    n, h, w, c, k, cout = shape
    d = _lib.ConvDesc(n, h, w, c, k, k, c, cout, 1, 1, 1, 1, 0, 0, accumulate, plan)
    if nbytes is not None:
        out = (C.c_int32 * 4)()
        assert L.axc_conv2d_route(table.handle, C.byref(d), nbytes, out) == 0
        return list(out)
    general, fast = C.c_size_t(), C.c_size_t()
    assert L.axc_conv2d_workspace_bytes(C.byref(d), C.byref(general)) == 0
    assert L.axc_conv2d_fast_workspace_bytes(table.handle, C.byref(d), C.byref(fast)) == 0
    return general.value, fast.value


@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_route_names_the_kernels_that_serve_the_call(built, shape):
    import tf_approximate_b200 as ax
    t = ax.Table(array=ax.noisy_table(3))
    general, scratch = ask(t, shape, 1)
    kind, tile, splits, in_global = ask(t, shape, 1, scratch)
    assert scratch > 0 and kind == EXPANDED and tile % 32 == 0 and 32 <= tile <= 2048 and (splits, in_global) == (1, 0)
    assert ask(t, shape, 1, scratch - 1)[0] == (COMMON_K if scratch - 1 >= general else NONE)
    # with a plan to keep: the plan's size leads to the kernel without expanded tables, the size that the query names to theirs
    both = ask(t, shape, 0)[1]
    assert both == (scratch if scratch < general else general + scratch)
    assert ask(t, shape, 0, both) == [EXPANDED, tile, 1, 0]
    assert ask(t, shape, 0, general)[0] == COMMON_K and ask(t, shape, 0, general + scratch)[0] == EXPANDED
    # a table with small entries: no partial sum rounds, and the route is that of the exact sum
    small = ax.Table(array=(ax.noisy_table(3) >> 8))
    assert ask(small, shape, 0, general)[0] == PLAN


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES, ids=["-".join(str(v) for v in s) for s in SHAPES])
def test_status_behind_a_kept_plan(built, shape):
    """The buffer's first part, where a plan would lie, holds neither a plan nor a header: a status read from there is not 0."""
    import torch
    import tf_approximate_b200 as ax
    n, h, w, c, k, cout = shape
    t = ax.Table(array=ax.noisy_table(3))
    general, scratch = ask(t, shape, 1)
    g = torch.Generator(device="cuda").manual_seed(3)
    x, f = torch.rand((n, h, w, c), device="cuda", generator=g), torch.randn((k, k, c, cout), device="cuda", generator=g) * 0.1
    args = (0.0, 1.0, -0.3, 0.4, [1, 1, 1, 1], 8, t, "SAME")
    want = ax.approx_conv2d_with_min_max_vars(x, f, *args, accumulate="reference")
    ws = torch.full((general + scratch,), 0x5A, dtype=torch.uint8, device="cuda")
    y, dbg = ax.approx_conv2d_with_min_max_vars(x, f, *args, accumulate="reference", workspace=ws, debug=True)
    assert dbg["plan"]["route"]["kernels"] == "expanded"
    assert (dbg["plan"]["rebuilt"], dbg["plan"]["fallback"], dbg["plan"]["status"], dbg["plan"]["steps_per_mille"]) == (0, 0, 0, 1000)
    assert torch.equal(y.view(torch.int32), want.view(torch.int32)) and bool((ws[:general] == 0x5A).all())
