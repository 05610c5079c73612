"""GPU: what the expanded-table kernels do when a wait inside them runs out.  The debug flavour lets a test set the limit to
nothing, for the kernel that makes the tables or for the convolution: the kernels must finish, the header must say 3, no
access may leave its bounds, and with the limit back the same calls must give the checker's bits again."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes as C, sys
import numpy as np, torch
sys.path.insert(0, %r)
import tf_approximate_b200 as ax
from tf_approximate_b200 import _lib
from oracle import oracle as O
L = _lib.load()
rec = (C.c_uint32 * 4)()
assert L.axc_debug_bounds_record(0, rec) == 0, "not the debug flavour"
rng = np.random.Generator(np.random.PCG64(8))
digits = rng.integers(0, 65280, 65536).astype(np.uint16)
# tables from global memory, and made by the CTAs with and without K split over CTAs; one-byte and two-digit entries, and an exact
# table, whose kernel has no such wait
for lut, waits in ((ax.truncated_table(), True), (digits, True), (ax.exact_table(), False)):
    t = ax.Table(array=lut)
    for n, h, w, c, k, co, in_global in ((4, 56, 57, 32, 3, 64, True), (2, 20, 20, 32, 3, 64, False), (1, 7, 7, 512, 1, 512, False)):
        x = rng.uniform(-1, 1, (n, h, w, c)).astype(np.float32)
        f = rng.normal(0, 0.1, (k, k, c, co)).astype(np.float32)
        mm = (-1.0, 1.0, float(f.min()), float(f.max()))
        xd, fd = torch.from_numpy(x).cuda(), torch.from_numpy(f).cuda()
        ref = O.conv2d(O.desc(n, h, w, c, k, k, co), lut, x, f, *mm, want=("out_exact",))["out_exact"]
        for expand, convolution in ((0, -1), (-1, 0), (0, 0), (-1, -1)):
            assert L.axc_debug_wait_polls(0, expand, convolution) == 0
            y, dbg = ax.approx_conv2d_with_min_max_vars(xd, fd, *mm, [1, 1, 1, 1], 8, t, "SAME", debug=True)
            torch.cuda.synchronize()
            assert dbg["plan"]["route"]["kernels"] == "expanded"
            assert dbg["plan"]["route"]["tables_in_global_memory"] == (in_global and waits), dbg["plan"]["route"]
            gave_up = waits and (convolution == 0 or (expand == 0 and in_global))
            assert dbg["plan"]["status"] == (3 if gave_up else 0), (lut[-1], n, h, expand, convolution, dbg["plan"])
            if not gave_up:
                assert np.array_equal(y.cpu().numpy().view(np.uint32), ref.view(np.uint32))
assert L.axc_debug_bounds_record(0, rec) == 0
print("violations", rec[0], "site", rec[1], "value", rec[2] | (rec[3] << 32))
assert rec[0] == 0
"""


@pytest.mark.gpu
def test_a_wait_that_runs_out_is_reported(built):
    env = dict(os.environ, AXC_LIBRARY_FLAVOUR="check")
    r = subprocess.run([sys.executable, "-c", CHILD % ROOT], env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
    assert "violations 0" in r.stdout


def test_normal_build_has_no_wait_limit_to_set(built):
    from tf_approximate_b200 import _lib
    assert _lib.load().axc_debug_wait_polls(0, 0, 0) == 12       # Unimplemented
