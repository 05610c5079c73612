"""Which kernels a call takes and how large its buffer must be is one decision: the size queries, the entry points' checks and
the launches agree, also with the environment switch AXC_DENSE_VARIANT=1 (the common-K kernel for every dense call).  The
switch is read once per process, so these tests run child processes; the refusals come before anything touches a device."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# n, h, w, c, k, cout: expanded tables smaller than the plan (filters much larger than the input), and larger
SHAPES = [(1, 7, 7, 512, 3, 512), (1, 14, 14, 256, 3, 256), (1, 7, 7, 2048, 1, 512), (8, 28, 28, 64, 3, 64)]

HEAD = r"""
import ctypes as C, sys
sys.path.insert(0, %r)
import tf_approximate_b200 as ax
from tf_approximate_b200 import _lib
L = _lib.load()
SHAPES = %r
def desc(n, h, w, c, k, cout, accumulate=0, plan=0):
    return _lib.ConvDesc(n, h, w, c, k, k, c, cout, 1, 1, 1, 1, 0, 0, accumulate, plan)
def size(fn, *args):
    b = C.c_size_t()
    assert fn(*args, C.byref(b)) == 0
    return b.value
""" % (ROOT, SHAPES)

SIZES = HEAD + r"""
t = ax.Table(array=ax.noisy_table(3))
for s in SHAPES:
    d = C.byref(desc(*s))
    print(size(L.axc_conv2d_fast_workspace_bytes, t.handle, d), size(L.axc_conv2d_workspace_bytes, d),
          size(L.axc_qconv2d_fast_workspace_bytes, t.handle, d), size(L.axc_qconv2d_workspace_bytes, d))
"""

REFUSED = HEAD + r"""
t = ax.Table(array=ax.noisy_table(3))
for s, (fast, general, qfast, qgeneral) in zip(SHAPES, %r):
    d = C.byref(desc(*s))
    assert size(L.axc_conv2d_fast_workspace_bytes, t.handle, d) == 0 and size(L.axc_conv2d_fast_workspace_bytes, None, d) == 0
    assert size(L.axc_qconv2d_fast_workspace_bytes, t.handle, d) == 0 and size(L.axc_qconv2d_fast_workspace_bytes, None, d) == 0
    for b in {fast, general - 1}:
        if b < general:
            assert L.axc_conv2d_forward(t.handle, d, 256, 256, 0.0, 1.0, 0.0, 1.0, 256, 256, b, None, 0, None) == 13, (s, b)
    for b in {qfast, qgeneral - 1}:
        if b < qgeneral:
            assert L.axc_qconv2d_forward(t.handle, d, 256, 256, 0, 0, 256, 256, b, 0, None) == 13, (s, b)
print("refused")
"""


def child(code, **env):
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, **env), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    return r.stdout


def default_sizes():
    env = {k: v for k, v in os.environ.items() if k != "AXC_DENSE_VARIANT"}
    r = subprocess.run([sys.executable, "-c", SIZES], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    return [tuple(int(v) for v in line.split()) for line in r.stdout.splitlines()]


def test_switch_to_the_common_k_kernel_needs_its_workspace(built):
    """With the switch set the queries offer no scratch of the expanded tables, and a buffer of that size - smaller than the
    common-K kernel's program - is refused by both entry points."""
    sizes = default_sizes()
    assert all(s[0] > 0 and s[2] > 0 for s in sizes)
    assert any(s[0] < s[1] for s in sizes) and any(s[2] < s[3] for s in sizes)
    assert "refused" in child(REFUSED % (sizes,), AXC_DENSE_VARIANT="1")


COMMON_K = HEAD + r"""
import numpy as np, torch
from oracle import oracle as O
rng = np.random.Generator(np.random.PCG64(9))
lut = ax.noisy_table(3)
t = ax.Table(array=lut)
for n, h, w, c, k, cout in SHAPES[:3]:
    x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
    f = rng.normal(0, 0.1, (k, k, c, cout)).astype(np.float32)
    mm = (-1.0, 1.0, float(f.min()), float(f.max()))
    ref = O.conv2d(O.desc(n, h, w, c, k, k, cout), lut, x, f, *mm, want=("out_exact", "acc"))
    y, dbg = ax.approx_conv2d_with_min_max_vars(torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda(), *mm, [1, 1, 1, 1], 8, t, "SAME", debug=True)
    assert dbg["plan"]["steps_per_mille"] == 0      # no plan, no expanded tables
    assert np.array_equal(dbg["acc"].cpu().numpy(), ref["acc"])
    assert np.array_equal(y.cpu().numpy().view(np.uint32), ref["out_exact"].view(np.uint32))
    a, b = rng.integers(0, 256, (n, h, w, c)).astype(np.uint8), rng.integers(0, 256, (k, k, c, cout)).astype(np.uint8)
    q, _, _ = ax.ax_conv2d(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), -1.0, 2.0, -0.5, 0.5, [1, 1, 1, 1], "SAME", table=t, ax_tune=False)
    want = O.qconv2d(O.desc(n, h, w, c, k, k, cout), lut, a, b, O.quantized_zero_point(-1.0, 2.0), O.quantized_zero_point(-0.5, 0.5))
    assert np.array_equal(q.cpu().numpy(), want)
print("served")
"""


@pytest.mark.gpu
def test_switch_to_the_common_k_kernel_serves_the_calls(built):
    assert "served" in child(COMMON_K, AXC_DENSE_VARIANT="1")


def routes(fn, table, shape, nbytes, plan):
    import ctypes as C
    from tf_approximate_b200 import _lib
    n, h, w, c, k, cout = shape
    out = (C.c_int32 * 4)()
    d = _lib.ConvDesc(n, h, w, c, k, k, c, cout, 1, 1, 1, 1, 0, 0, 0, plan)
    assert getattr(_lib.load(), fn)(table.handle, C.byref(d), nbytes, out) == 0
    return out[0]


def sizes(fn, table, shape, plan):
    import ctypes as C
    from tf_approximate_b200 import _lib
    n, h, w, c, k, cout = shape
    b = C.c_size_t()
    d = _lib.ConvDesc(n, h, w, c, k, k, c, cout, 1, 1, 1, 1, 0, 0, 0, plan)
    args = (C.byref(d), C.byref(b)) if table is None else (table.handle, C.byref(d), C.byref(b))
    assert getattr(_lib.load(), fn)(*args) == 0
    return b.value


@pytest.mark.parametrize("op", ["axc_conv2d", "axc_qconv2d"])
@pytest.mark.parametrize("layer", [(7, 7, 512, 3, 512), (28, 28, 64, 3, 64), (14, 14, 256, 1, 1024)])
def test_a_buffer_that_can_hold_a_plan_is_the_plans(built, op, layer):
    """A kept buffer of the documented size goes to the plan whatever the batch; the sizes that the queries name for the
    expanded tables lead there, one byte less does not; and with no plan to keep their scratch alone is enough."""
    import tf_approximate_b200 as ax
    NONE, PLAN, COMMON_K, EXPANDED = range(4)
    t = ax.Table(array=ax.noisy_table(3))
    below = above = 0
    for n in (1, 2, 8, 64, 128, 256):
        s = (n,) + layer
        general, keep, none = sizes(op + "_workspace_bytes", None, s, 0), sizes(op + "_fast_workspace_bytes", t, s, 0), sizes(op + "_fast_workspace_bytes", t, s, 1)
        assert routes(op + "_route", t, s, general, 0) == PLAN and none > 0
        below += none < general
        above += none >= general
        assert keep == (none if none < general else general + none)
        assert routes(op + "_route", t, s, keep, 0) == EXPANDED and routes(op + "_route", t, s, none, 1) == EXPANDED
        assert routes(op + "_route", t, s, keep - 1, 0) == (NONE if keep < general else PLAN)
        assert routes(op + "_route", t, s, none - 1, 1) == (NONE if none - 1 < general else COMMON_K)
    assert above or op == "axc_qconv2d"
    assert below or layer != (7, 7, 512, 3, 512)


@pytest.mark.gpu
def test_a_kept_plan_survives_every_batch_size(built):
    """One buffer per layer, called with full and ragged batches and with device ranges: the plan is built once.  A buffer with
    room for the expanded tables behind the plan takes them and leaves the plan alone."""
    import ctypes as C
    import torch
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import _lib, ops
    g = torch.Generator(device="cuda").manual_seed(6)
    t = ax.Table(array=ax.noisy_table(4))
    f = torch.randn((3, 3, 128, 128), device="cuda", generator=g) * 0.05
    one = [1, 1, 1, 1]
    plan_bytes = ops.workspace_bytes((1, 7, 7, 128), f.shape, one, "SAME")
    both = ops.fast_workspace_bytes((128, 7, 7, 128), f.shape, one, "SAME", table=t, plan="keep")
    assert both > plan_bytes
    for size, last in ((plan_bytes, "plan"), (both, "expanded")):
        ws = torch.zeros(size, dtype=torch.uint8, device="cuda")
        rebuilt = []
        for n in (8, 64, 128, 8):
            x = torch.rand((n, 7, 7, 128), device="cuda", generator=g) * 2 - 1
            y, dbg = ax.approx_conv2d_with_min_max_vars(x, f, -1.0, 1.0, -0.2, 0.2, one, 8, t, "SAME", workspace=ws, debug=True)
            assert dbg["plan"]["status"] == 0
            if n == 128:
                assert dbg["plan"]["route"]["kernels"] == last
            if dbg["plan"]["route"]["kernels"] == "expanded":
                assert dbg["plan"]["steps_per_mille"] == 1000 and dbg["plan"]["rebuilt"] == 0
            if dbg["plan"]["route"]["kernels"] == "plan":
                rebuilt.append(dbg["plan"]["rebuilt"])
            want = ax.approx_conv2d_with_min_max_vars(x, f, -1.0, 1.0, -0.2, 0.2, one, 8, t, "SAME")
            assert torch.equal(y.view(torch.int32), want.view(torch.int32))
        assert rebuilt[:1] in ([1], []) and not any(rebuilt[1:])
        if size == plan_bytes:
            assert rebuilt == [1, 0, 0, 0]
    # the quantised entry point keeps the plan in the same place
    L = _lib.load()
    ws, word = None, (C.c_int32 * 4)()
    b = torch.randint(0, 256, (3, 3, 128, 128), device="cuda", generator=g, dtype=torch.uint8)
    zero = [C.c_int32(), C.c_int32()]
    assert L.axc_quantized_zero_point(-1.0, 2.0, C.byref(zero[0])) == 0 and L.axc_quantized_zero_point(-0.5, 0.5, C.byref(zero[1])) == 0
    rebuilt = []
    for n in (128, 8, 128):
        a = torch.randint(0, 256, (n, 7, 7, 128), device="cuda", generator=g, dtype=torch.uint8)
        d = _lib.ConvDesc(n, 7, 7, 128, 3, 3, 128, 128, 1, 1, 1, 1, 0, 0, 0, 0)
        if ws is None:
            need = C.c_size_t()
            assert L.axc_qconv2d_workspace_bytes(C.byref(d), C.byref(need)) == 0
            ws = torch.zeros(need.value, dtype=torch.uint8, device="cuda")
        y = torch.empty((n, 7, 7, 128), dtype=torch.int32, device="cuda")
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert L.axc_qconv2d_forward(t.handle, C.byref(d), a.data_ptr(), b.data_ptr(), zero[0].value, zero[1].value, y.data_ptr(), ws.data_ptr(),
                                     sizes("axc_qconv2d_workspace_bytes", None, (n, 7, 7, 128, 3, 128), 0), 0, stream) == 0
        assert L.axc_conv2d_plan_info(ws.data_ptr(), word, 0, stream) == 0
        rebuilt.append(word[0])
        want, _, _ = ax.ax_conv2d(a, b, -1.0, 2.0, -0.5, 0.5, one, "SAME", table=t, ax_tune=False)
        assert torch.equal(y, want)
    assert rebuilt == [1, 0, 0]


@pytest.mark.gpu
def test_a_device_without_room_for_the_scratch_still_serves_the_call(built, monkeypatch):
    """Where the expanded tables' scratch cannot be allocated the call runs on the kernels that need a plan's workspace only:
    same bits, no error - the op, the layer-level caller, the quantised op and the sharded call."""
    import torch
    import tf_approximate_b200 as ax
    from tf_approximate_b200 import parallel
    g = torch.Generator(device="cuda").manual_seed(12)
    t = ax.Table(array=ax.noisy_table(6))
    x = torch.rand((8, 28, 28, 64), device="cuda", generator=g)
    f = torch.randn((3, 3, 64, 64), device="cuda", generator=g) * 0.1
    a = torch.randint(0, 256, x.shape, device="cuda", generator=g, dtype=torch.uint8)
    b = torch.randint(0, 256, f.shape, device="cuda", generator=g, dtype=torch.uint8)
    layer = ax.FakeApproxConv2D(64, 64, 3, padding="same", mul_map_file=t).cuda().eval()
    one = [1, 1, 1, 1]

    def calls():
        with torch.no_grad():
            return [ax.approx_conv2d_with_min_max_vars(x, f, 0.0, 1.0, -0.4, 0.4, one, 8, t, "SAME"), layer(x),
                    ax.ax_conv2d(a, b, -1.0, 2.0, -0.5, 0.5, one, "SAME", table=t, ax_tune=False)[0],
                    parallel.forward_sharded([x[:5], x[5:]], [f, f], t, (0.0, 1.0, -0.4, 0.4), one, "SAME", gather_to="cuda:0")]
    want = calls()
    empty, refused = torch.empty, []

    def full(*args, **kw):
        if kw.get("dtype") == torch.uint8:
            refused.append(args)
            raise torch.OutOfMemoryError("out of memory")
        return empty(*args, **kw)
    monkeypatch.setattr(torch, "empty", full)
    got = calls()
    monkeypatch.undo()
    assert len(refused) == 5
    for w, y in zip(want, got):
        assert torch.equal(w.view(torch.int32), y.view(torch.int32))
