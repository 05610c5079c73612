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
